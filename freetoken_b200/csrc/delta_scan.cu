#include "delta_scan.cuh"

using namespace ft;

// The gated delta rule with one decay per head.
extern "C" int ft_delta_scan(const void* qkv, long long ld, const void* beta, const void* decay, long long ld_gate,
                  const float* dt_bias, const float* A_log, float* state, long long slot_stride, float* o,
                  const int* seg_slot, const int* seg_q_start, int heads, int P, int D, int G, float unit_eps,
                  float q_scale, int S, int T, int longest, int dtype,
                  int state_ahead, cudaStream_t stream) {
  if (S <= 0) return FT_OK;
  if (heads <= 0 || P <= 0 || D <= 0 || D > 256 || G <= 0 || heads % G) return FT_ERR_SHAPE;
  DeltaArgs a{qkv, beta, decay, dt_bias, A_log, state, o, seg_slot, seg_q_start, ld, ld_gate, slot_stride,
              heads, P, D, G, unit_eps, q_scale, 0, nullptr, 0, nullptr, nullptr, 0, state_ahead};
  return dispatch_delta<0>(a, S, T, longest, dtype, stream);
}

FT_PACKED(ft_delta_scan)
