#include "delta_scan.cuh"

using namespace ft;

// The delta rule with a decay per key channel: `decay` is float32 [T, ld_decay] (channel n of head
// h at column h * D + n), dt_bias [heads * D].
extern "C" int ft_channel_delta_scan(const void* qkv, long long ld, const void* beta, long long ld_gate, const float* decay,
                          long long ld_decay, const float* dt_bias, const float* A_log, float* state,
                          long long slot_stride, float* o, const int* seg_slot, const int* seg_q_start, int heads,
                          int P, int D, int G, float unit_eps, float q_scale, int S, int T, int longest, int dtype,
                  int state_ahead, cudaStream_t stream) {
  if (S <= 0) return FT_OK;
  if (heads <= 0 || P <= 0 || D <= 0 || D > 256 || G <= 0 || heads % G) return FT_ERR_SHAPE;
  DeltaArgs a{qkv, beta, nullptr, dt_bias, A_log, state, o, seg_slot, seg_q_start, ld, ld_gate, slot_stride,
              heads, P, D, G, unit_eps, q_scale, 0, decay, ld_decay, nullptr, nullptr, 0, state_ahead};
  return dispatch_delta<1>(a, S, T, longest, dtype, stream);
}

FT_PACKED(ft_channel_delta_scan)
