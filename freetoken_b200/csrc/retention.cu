#include "delta_scan.cuh"

using namespace ft;

// Retention: rows of `qkv` are q (heads * D) | k (heads * D) | v (heads * P); `decay` [heads] float32 holds
// each head's constant factor; cos_sin [positions, rot_dims] (rot_dims 0: nothing turns).
extern "C" int ft_retention_scan(const void* qkv, long long ld, const float* decay, const float* cos_sin, int rot_dims,
                      const int* seg_pos0, float* state, long long slot_stride, float* o, const int* seg_slot,
                      const int* seg_q_start, int heads, int P, int D, float k_scale, int S, int T, int longest, int dtype,
                  int state_ahead, cudaStream_t stream) {
  if (S <= 0) return FT_OK;
  if (heads <= 0 || P <= 0 || D <= 0 || D > 256 || rot_dims < 0 || (rot_dims & 1) || rot_dims > D)
    return FT_ERR_SHAPE;
  DeltaArgs a{qkv, nullptr, nullptr, decay, nullptr, state, o, seg_slot, seg_q_start, ld, 0, slot_stride,
              heads, P, D, heads, 0.f, k_scale, 0, nullptr, 0, cos_sin, seg_pos0, cos_sin ? rot_dims : 0, state_ahead};
  return dispatch_delta<2>(a, S, T, longest, dtype, stream);
}

FT_PACKED(ft_retention_scan)
