// The gated delta rule, the same with a decay per key channel, and retention: three modes of the same kernels, each compiled
// in a library of its own (delta_scan.cu, channel_delta.cu, retention.cu).
//
//   delta_scan       S <- g S ; u = beta (v - S^T k) ; S <- S + k u^T ; o = S^T q   (S: D x P per head)
//
// State layout, lanes and columns: scans.cuh.
#pragma once
#include "scans.cuh"

namespace ft {

struct DeltaArgs {
  const void* qkv;      // [T, ld]: q (G * D) | k (G * D) | v (heads * P), after convolution and silu
  const void* beta;     // [T, ld_gate]: the write strength's projection, head h at column h
  const void* decay;    // [T, ld_gate]: the decay's projection, head h at column h
  const float* dt_bias; // [heads]
  const float* A_log;   // [heads]
  float* state;         // slot s: state + s * slot_stride, [heads][D][P]
  float* o;             // [T, heads * P] float32
  const int* seg_slot;
  const int* seg_q_start;
  long long ld, ld_gate, slot_stride;
  int heads, P, D, G;
  float unit_eps, q_scale;
  int vec;
  // MODE 1: a decay per key channel
  const float* decay_rows;   // [T, ld_decay] float32: the decay's projection, channel n of head h at h * D + n;
  long long ld_decay;        // dt_bias is then [heads * D]
  // MODE 2: retention
  const float* cos_sin;      // [positions, rot_dims]: cos | sin (nullptr or rot_dims 0: no rotation)
  const int* seg_pos0;       // [S]: position of a segment's first token
  int rot_dims;
  int state_ahead;           // the launch right in front does not write the state: it is fetched ahead of the wait
};

// MODE 0: the gated delta rule with one decay per head.
// MODE 1: the same rule with a decay per key channel: row n of a head's state is multiplied by
//         g_n = exp(-exp(A_log_h) softplus(a_n + dt_bias[h * D + n])) before the token reads and writes.
// MODE 2: retention: S <- c_h S + k v^T, o = S^T q with a constant c_h per head (dt_bias[h]), no write
//         strength and no unit norms; q and k have the first rot_dims dimensions of each head turned
//         by the token's position (dimension i with i + rot_dims / 2) in shared memory, in float32;
//         k is multiplied by q_scale after the rotation.
// CH: tokens of a chunk.  Segments of one token each take a chunk of one: the rows staged for a chunk of eight took
// registers that left four requests of 32 heads of 128 x 128 two rounds of blocks.
template <typename AT, int NPL, int WC, int MODE, int CH>
__global__ void __launch_bounds__(SCAN_THREADS) delta_scan_kernel(DeltaArgs a) {
  constexpr int COLS = SCAN_WARPS * WC;
  constexpr int NB = (NPL * 32 + SCAN_THREADS - 1) / SCAN_THREADS;
  constexpr int XR = (CH * COLS + SCAN_THREADS - 1) / SCAN_THREADS;
  extern __shared__ float sm[];
  if (!a.state_ahead) pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int head = blockIdx.y, seg = blockIdx.z;
  const int D = a.D, P = a.P;
  const int g = head / (a.heads / a.G);
  const int col0 = blockIdx.x * COLS;
  const int j0 = col0 + warp * WC;
  const int width = a.heads * P;
  const int per = CH * ((MODE == 1 ? 3 : 2) * D + COLS + 2);
  const int q0 = a.seg_q_start[seg], q1 = a.seg_q_start[seg + 1];
  float* st = a.state + (size_t)a.seg_slot[seg] * a.slot_stride + (size_t)head * D * P;
  const float rate = MODE == 2 ? 0.f : -expf(a.A_log[head]);
  const float bias = MODE == 1 ? 0.f : a.dt_bias[head];      // MODE 2: the head's constant decay
  const AT* qkv = (const AT*)a.qkv;
  const int half = MODE == 2 ? a.rot_dims >> 1 : 0;
  const int pos0 = MODE == 2 && half ? a.seg_pos0[seg] : 0;
  float ch_bias[NB];                                          // MODE 1: dt_bias of this thread's channels
  if constexpr (MODE == 1) {
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const int n = threadIdx.x + SCAN_THREADS * b;
      ch_bias[b] = n < D ? a.dt_bias[(size_t)head * D + n] : 0.f;
    }
  }

  float S[NPL][WC];
#pragma unroll
  for (int e = 0; e < NPL; ++e) {
    const int n = lane + 32 * e;
    if (n < D) load_cols<WC>(st + (size_t)n * P + j0, S[e], P - j0, a.vec);
    else {
#pragma unroll
      for (int c = 0; c < WC; ++c) S[e][c] = 0.f;
    }
  }
  if (a.state_ahead) pdl_wait();

  AT pq[CH][NB], pk[CH][NB], pv[XR], pbeta, pdecay;
  float pg[MODE == 1 ? CH : 1][NB];                   // MODE 1: the channels' decay projections
  float pcos[MODE == 2 ? NPL : 1], psin[MODE == 2 ? NPL : 1]; // MODE 2: pair (tt, i) = threadIdx.x + 128 r
  auto fetch = [&](int t0, int nt) {
#pragma unroll
    for (int tt = 0; tt < CH; ++tt) {
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int n = threadIdx.x + SCAN_THREADS * b;
        if (tt < nt && n < D) {
          const AT* row = qkv + (size_t)(t0 + tt) * a.ld + (size_t)g * D + n;
          pq[tt][b] = row[0];
          pk[tt][b] = row[(size_t)a.G * D];
          if constexpr (MODE == 1) pg[tt][b] = a.decay_rows[(size_t)(t0 + tt) * a.ld_decay + (size_t)head * D + n];
        }
      }
    }
    if constexpr (MODE == 2) {
#pragma unroll
      for (int r = 0; r < NPL; ++r) {
        const int idx = threadIdx.x + SCAN_THREADS * r;
        if (half && idx < nt * half) {
          const int tt = idx / half, i = idx - tt * half;
          const float* cs = a.cos_sin + (size_t)(pos0 + t0 + tt - q0) * a.rot_dims;
          pcos[r] = cs[i];
          psin[r] = cs[half + i];
        }
      }
    }
#pragma unroll
    for (int r = 0; r < XR; ++r) {
      const int i = threadIdx.x + SCAN_THREADS * r, tt = i / COLS, c = i % COLS;
      pv[r] = (tt < nt && col0 + c < P)
                  ? qkv[(size_t)(t0 + tt) * a.ld + 2 * (size_t)a.G * D + (size_t)head * P + col0 + c]
                  : from_float<AT>(0.f);
    }
    if (MODE != 2 && (int)threadIdx.x < nt) {
      const size_t at = (size_t)(t0 + threadIdx.x) * a.ld_gate + head;
      pbeta = ((const AT*)a.beta)[at];
      if constexpr (MODE == 0) pdecay = ((const AT*)a.decay)[at];
    }
  };
  auto put = [&](float* buf, int nt) {
    float* qs = buf;
    float* ks = qs + CH * D;
    float* vs = ks + CH * D;
    float* gates = vs + CH * COLS;
#pragma unroll
    for (int tt = 0; tt < CH; ++tt) {
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int n = threadIdx.x + SCAN_THREADS * b;
        if (tt < nt && n < D) {
          qs[tt * D + n] = to_float(pq[tt][b]);
          ks[tt * D + n] = to_float(pk[tt][b]);
          if constexpr (MODE == 1)
            gates[2 * CH + tt * D + n] = expf(rate * softplus_f(pg[tt][b] + ch_bias[b]));
        }
      }
    }
#pragma unroll
    for (int r = 0; r < XR; ++r) {
      const int i = threadIdx.x + SCAN_THREADS * r;
      if (i < CH * COLS) vs[i] = to_float(pv[r]);
    }
    if ((int)threadIdx.x < nt) {
      if constexpr (MODE == 2) {
        gates[threadIdx.x] = 1.f;
        gates[CH + threadIdx.x] = bias;
      } else {
        gates[threadIdx.x] = 1.f / (1.f + expf(-to_float(pbeta)));
        gates[CH + threadIdx.x] = MODE == 1 ? 1.f : expf(rate * softplus_f(to_float(pdecay) + bias));
      }
    }
  };
  // MODE 2: turn the staged q and k rows of a chunk; a thread owns whole pairs
  auto turn_rows = [&](float* buf, int nt) {
    if constexpr (MODE == 2) {
      float* qs = buf;
      float* ks = qs + CH * D;
#pragma unroll
      for (int r = 0; r < NPL; ++r) {
        const int idx = threadIdx.x + SCAN_THREADS * r;
        if (half && idx < nt * half) {
          const int tt = idx / half, i = idx - tt * half;
          const float c = pcos[r], sn = psin[r];
          float* qa = qs + tt * D + i;
          float* ka = ks + tt * D + i;
          const float qu = qa[0], qv = qa[half], ku = ka[0], kv_ = ka[half];
          qa[0] = qu * c - qv * sn;
          qa[half] = qv * c + qu * sn;
          ka[0] = ku * c - kv_ * sn;
          ka[half] = kv_ * c + ku * sn;
        }
      }
    }
  };

  fetch(q0, min(CH, q1 - q0));
  put(sm, min(CH, q1 - q0));
  if constexpr (MODE == 2) {
    __syncthreads();
    turn_rows(sm, min(CH, q1 - q0));
  }
  __syncthreads();
  int turn = 0;
  for (int t0 = q0; t0 < q1; t0 += CH, turn ^= 1) {
    const int nt = min(CH, q1 - t0);
    const int next = min(CH, q1 - t0 - CH);
    if (next > 0) fetch(t0 + CH, next);
    const float* qs = sm + turn * per;
    const float* ks = qs + CH * D;
    const float* vs = ks + CH * D;
    const float* gates = vs + CH * COLS;
    auto token = [&](int tt) {
      const float beta = gates[tt], decay = gates[CH + tt];
      float qv[NPL], kv[NPL];
      // sums of squares of the raw q and k rows and their product: unit vectors without a pass of
      // their own (every warp of the block forms them for itself; they do not wait for the state)
      float unit[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int e = 0; e < NPL; ++e) {
        const int n = lane + 32 * e;
        qv[e] = n < D ? qs[tt * D + n] : 0.f;
        kv[e] = n < D ? ks[tt * D + n] : 0.f;
        if constexpr (MODE == 2) kv[e] *= a.q_scale;
        unit[0] = fmaf(qv[e], qv[e], unit[0]);
        unit[1] = fmaf(kv[e], kv[e], unit[1]);
        unit[2] = fmaf(qv[e], kv[e], unit[2]);
      }
      warp_sum_multi<4>(unit);
      const float mine_u = unit[0];                       // lane l holds value l >> 3
      float kq;
      if constexpr (MODE == 2) {
        kq = __shfl_sync(0xffffffffu, mine_u, 16);
      } else {
        const float iq = a.q_scale / sqrtf(__shfl_sync(0xffffffffu, mine_u, 0) + a.unit_eps);
        const float ik = 1.f / sqrtf(__shfl_sync(0xffffffffu, mine_u, 8) + a.unit_eps);
        kq = __shfl_sync(0xffffffffu, mine_u, 16) * iq * ik;
#pragma unroll
        for (int e = 0; e < NPL; ++e) {
          qv[e] *= iq;
          kv[e] *= ik;
        }
      }
      if constexpr (MODE == 1) {
        // every row of the state decays by its own channel's factor before the token reads it
#pragma unroll
        for (int e = 0; e < NPL; ++e) {
          const int n = lane + 32 * e;
          const float gn = n < D ? gates[2 * CH + tt * D + n] : 1.f;
#pragma unroll
          for (int c = 0; c < WC; ++c) S[e][c] *= gn;
        }
      }
      // per column: S^T k and S^T q of the state before this token
      float red[2 * WC];
#pragma unroll
      for (int c = 0; c < WC; ++c) {
        float sa = 0.f, sb = 0.f;
#pragma unroll
        for (int e = 0; e < NPL; ++e) {
          sa = fmaf(S[e][c], kv[e], sa);
          sb = fmaf(S[e][c], qv[e], sb);
        }
        red[c] = sa;
        red[WC + c] = sb;
      }
      warp_sum_multi<2 * WC>(red);
      constexpr int SHIFT = 5 - Log2<2 * WC>::value;      // lane l holds the total of value l >> SHIFT
      const float mine = red[0];
#pragma unroll
      for (int c = 0; c < WC; ++c) {
        const float sa = __shfl_sync(0xffffffffu, mine, c << SHIFT);
        const float sb = __shfl_sync(0xffffffffu, mine, (WC + c) << SHIFT);
        const float v = vs[tt * COLS + warp * WC + c];
        // the decayed state answers k with decay * sa; the token writes u along k, and its own
        // read-out already contains that write: decay * sb + (k . q) u
        const float u = MODE == 2 ? v : beta * (v - decay * sa);
        if (lane == 0 && j0 + c < P)
          a.o[(size_t)(t0 + tt) * width + (size_t)head * P + j0 + c] = fmaf(kq, u, decay * sb);
#pragma unroll
        for (int e = 0; e < NPL; ++e) S[e][c] = fmaf(kv[e], u, decay * S[e][c]);
      }
    };
    if (nt == CH) {
#pragma unroll
      for (int tt = 0; tt < CH; ++tt) token(tt);
    } else {
      for (int tt = 0; tt < nt; ++tt) token(tt);
    }
    if (next > 0) put(sm + (turn ^ 1) * per, next);
    if constexpr (MODE == 2) {
      if (next > 0) {
        __syncthreads();
        turn_rows(sm + (turn ^ 1) * per, next);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int e = 0; e < NPL; ++e) {
    const int n = lane + 32 * e;
    if (n < D) store_cols<WC>(st + (size_t)n * P + j0, S[e], P - j0, a.vec);
  }
}

// The three modes of delta_scan_kernel.
template <typename AT, int NPL, int CPL, int MODE>
__global__ void __launch_bounds__(SEQ_THREADS, NPL < 8 ? 2 : 1) delta_seq_kernel(DeltaArgs a) {
  constexpr int R = 2 * NPL, DP = 32 * NPL, COLS = 2 * SEQ_WARPS * CPL;
  constexpr int PER = seq_buffer(NPL, CPL, MODE == 1 ? 3 : 2);
  constexpr int VR = (SEQ_CHUNK * COLS + 32 * SEQ_WARPS - 1) / (32 * SEQ_WARPS);
  extern __shared__ __align__(16) float sm[];
  // what a token writes, for its read-out: words of their own, since lanes behind the one that stores may still have to
  // read the token's value (retention writes the value itself)
  __shared__ float us[MODE == 2 ? 1 : SEQ_CHUNK * COLS];
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % SEQ_WARPS, l = lane & 15;
  const bool stages = threadIdx.x >= 32 * SEQ_WARPS;
  const int head = blockIdx.y, seg = blockIdx.z;
  const int D = a.D, P = a.P;
  const int q0 = a.seg_q_start[seg], q1 = a.seg_q_start[seg + 1];
  if (q1 <= q0) return;
  const int g = head / (a.heads / a.G);
  const int width = a.heads * P;
  const int col0 = blockIdx.x * COLS, cb = (2 * warp + (lane >> 4)) * CPL, col = col0 + cb;
  float* st = a.state + (size_t)a.seg_slot[seg] * a.slot_stride + (size_t)head * D * P;
  const float rate = MODE == 2 ? 0.f : -expf(a.A_log[head]);
  const float bias = MODE == 1 ? 0.f : a.dt_bias[head];          // MODE 2: the head's constant decay
  const AT* qkv = (const AT*)a.qkv;
  const int half = MODE == 2 ? a.rot_dims >> 1 : 0;
  const int pos0 = MODE == 2 && half ? a.seg_pos0[seg] : 0;
  float ch_bias[NPL];
  if constexpr (MODE == 1) {
#pragma unroll
    for (int e = 0; e < NPL; ++e) {
      const int n = lane + 32 * e;
      ch_bias[e] = n < D ? a.dt_bias[(size_t)head * D + n] : 0.f;
    }
  }
  struct Staged {
    AT q[SEQ_PER_WARP][NPL], k[SEQ_PER_WARP][NPL], v[VR], beta[SEQ_PER_WARP], decay[SEQ_PER_WARP];
    float g[MODE == 1 ? SEQ_PER_WARP : 1][NPL], c[MODE == 2 ? SEQ_PER_WARP : 1][NPL], s[MODE == 2 ? SEQ_PER_WARP : 1][NPL];
  } even, odd;
  auto fetch = [&](int t0, Staged& x) {
    const int nt = min(SEQ_CHUNK, q1 - t0);                      // may be 0 or less: nothing is read
#pragma unroll
    for (int j = 0; j < SEQ_PER_WARP; ++j) {
      const int tt = warp + SEQ_WARPS * j;
      const size_t t = t0 + tt;
#pragma unroll
      for (int e = 0; e < NPL; ++e) {
        const int n = lane + 32 * e;
        const bool in = tt < nt && n < D;
        const AT* row = qkv + t * a.ld + (size_t)g * D + n;
        x.q[j][e] = in ? row[0] : from_float<AT>(0.f);
        x.k[j][e] = in ? row[(size_t)a.G * D] : from_float<AT>(0.f);
        if constexpr (MODE == 1) x.g[j][e] = in ? a.decay_rows[t * a.ld_decay + (size_t)head * D + n] : 0.f;
        if constexpr (MODE == 2) {
          if (in && n < 2 * half) {
            const float* cs = a.cos_sin + (size_t)(pos0 + t0 + tt - q0) * a.rot_dims + (n < half ? n : n - half);
            x.c[j][e] = cs[0];
            x.s[j][e] = cs[half];
          }
        }
      }
      if (MODE != 2 && tt < nt) {
        const size_t at = t * a.ld_gate + head;
        x.beta[j] = ((const AT*)a.beta)[at];
        if constexpr (MODE == 0) x.decay[j] = ((const AT*)a.decay)[at];
      }
    }
#pragma unroll
    for (int r = 0; r < VR; ++r) {
      const int i = threadIdx.x % (32 * SEQ_WARPS) + 32 * SEQ_WARPS * r, tt = i / COLS, c = i % COLS;
      x.v[r] = (tt < nt && col0 + c < P)
                   ? qkv[(size_t)(t0 + tt) * a.ld + 2 * (size_t)a.G * D + (size_t)head * P + col0 + c]
                   : from_float<AT>(0.f);
    }
  };
  auto put = [&](float* buf, const Staged& x) {
    float* qs = buf;
    float* ks = qs + SEQ_CHUNK * DP;
    float* gs = ks + SEQ_CHUNK * DP;                             // MODE 1
    float* vs = gs + (MODE == 1 ? SEQ_CHUNK * DP : 0);
    float4* gates = reinterpret_cast<float4*>(vs + SEQ_CHUNK * COLS);      // write strength, decay, k . q
    float kq[SEQ_PER_WARP];
#pragma unroll
    for (int j = 0; j < SEQ_PER_WARP; ++j) {
      const int tt = warp + SEQ_WARPS * j;
      float qv[NPL], kv[NPL], unit[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int e = 0; e < NPL; ++e) {
        qv[e] = to_float(x.q[j][e]);
        kv[e] = to_float(x.k[j][e]);
      }
      if constexpr (MODE == 2) {
        if (half) {                                              // a pair's two values meet in the token's own rows
          float* qr = qs + tt * DP;
          float* kr = ks + tt * DP;
#pragma unroll
          for (int e = 0; e < NPL; ++e) {
            qr[lane + 32 * e] = qv[e];
            kr[lane + 32 * e] = kv[e];
          }
          __syncwarp();
#pragma unroll
          for (int e = 0; e < NPL; ++e) {
            const int n = lane + 32 * e;
            if (n < 2 * half) {                                  // rounded as delta_scan_kernel rounds
              const float c = x.c[j][e], sn = x.s[j][e];
              const int other = n < half ? n + half : n - half;
              const float qo = qr[other], ko = kr[other];
              qv[e] = n < half ? __fmaf_rn(qv[e], c, -__fmul_rn(qo, sn)) : __fmaf_rn(qo, sn, __fmul_rn(qv[e], c));
              kv[e] = n < half ? __fmaf_rn(kv[e], c, -__fmul_rn(ko, sn)) : __fmaf_rn(ko, sn, __fmul_rn(kv[e], c));
            }
          }
          __syncwarp();
        }
#pragma unroll
        for (int e = 0; e < NPL; ++e) kv[e] *= a.q_scale;
      }
#pragma unroll
      for (int e = 0; e < NPL; ++e) {
        unit[0] = fmaf(qv[e], qv[e], unit[0]);
        unit[1] = fmaf(kv[e], kv[e], unit[1]);
        unit[2] = fmaf(qv[e], kv[e], unit[2]);
      }
      warp_sum_multi<4>(unit);                                   // lane n holds value n >> 3
      if constexpr (MODE == 2) {
        kq[j] = __shfl_sync(0xffffffffu, unit[0], 16);
      } else {
        const float iq = a.q_scale / sqrtf(__shfl_sync(0xffffffffu, unit[0], 0) + a.unit_eps);
        const float ik = 1.f / sqrtf(__shfl_sync(0xffffffffu, unit[0], 8) + a.unit_eps);
        kq[j] = __shfl_sync(0xffffffffu, unit[0], 16) * iq * ik;
#pragma unroll
        for (int e = 0; e < NPL; ++e) {
          qv[e] *= iq;
          kv[e] *= ik;
        }
      }
#pragma unroll
      for (int e = 0; e < NPL; ++e) {
        const int n = lane + 32 * e, at = tt * DP + seq_place<NPL>(n);
        qs[at] = qv[e];
        ks[at] = kv[e];
        if constexpr (MODE == 1) gs[at] = n < D ? expf(rate * softplus_f(x.g[j][e] + ch_bias[e])) : 1.f;
      }
    }
    if (lane < SEQ_PER_WARP) {                                   // a lane a token
      float beta = 1.f, decay = bias, product = kq[0];
      if constexpr (MODE != 2) {
        AT raw_beta = x.beta[0], raw_decay = x.decay[0];
#pragma unroll
        for (int j = 1; j < SEQ_PER_WARP; ++j)
          if (lane == j) { raw_beta = x.beta[j]; raw_decay = x.decay[j]; }
        beta = 1.f / (1.f + expf(-to_float(raw_beta)));
        decay = MODE == 1 ? 1.f : expf(rate * softplus_f(to_float(raw_decay) + bias));
      }
#pragma unroll
      for (int j = 1; j < SEQ_PER_WARP; ++j)
        if (lane == j) product = kq[j];
      gates[warp + SEQ_WARPS * lane] = make_float4(beta, decay, product, 0.f);
    }
#pragma unroll
    for (int r = 0; r < VR; ++r) {
      const int i = threadIdx.x % (32 * SEQ_WARPS) + 32 * SEQ_WARPS * r;
      if (i < SEQ_CHUNK * COLS) vs[i] = to_float(x.v[r]);
    }
  };

  if (stages) {
    // two chunks on their way in registers; a buffer is filled while the other one is worked through
    fetch(q0, even);
    fetch(q0 + SEQ_CHUNK, odd);
    put(sm, even);
    fetch(q0 + 2 * SEQ_CHUNK, even);
    __syncthreads();
    for (int t0 = q0; t0 < q1; t0 += 2 * SEQ_CHUNK) {
      if (t0 + SEQ_CHUNK < q1) put(sm + PER, odd);
      fetch(t0 + 3 * SEQ_CHUNK, odd);
      __syncthreads();
      if (t0 + SEQ_CHUNK >= q1) break;
      if (t0 + 2 * SEQ_CHUNK < q1) put(sm, even);
      fetch(t0 + 4 * SEQ_CHUNK, even);
      __syncthreads();
    }
    return;
  }
  float S[R][CPL];
  seq_load_state<NPL, CPL>(st, D, P, col, l, a.vec, S);
  auto chunk = [&](int t0, int turn) {
    const int nt = min(SEQ_CHUNK, q1 - t0);
    const float* qs = sm + turn * PER;
    const float* ks = qs + SEQ_CHUNK * DP;
    const float* gs = ks + SEQ_CHUNK * DP;
    const float* vs = sm + turn * PER + (MODE == 1 ? 3 : 2) * SEQ_CHUNK * DP;
    const float4* gates = reinterpret_cast<const float4*>(vs + SEQ_CHUNK * COLS);
    float part[CPL][SEQ_CHUNK];
    auto token = [&](int tt) {
      float q[R], k[R], v[CPL];
      seq_row<NPL>(qs + tt * DP, l, q);
      seq_row<NPL>(ks + tt * DP, l, k);
      const float4 gate = gates[tt];
      if constexpr (MODE == 1) {
        float gn[R];
        seq_row<NPL>(gs + tt * DP, l, gn);
#pragma unroll
        for (int i = 0; i < R; ++i)
#pragma unroll
          for (int c = 0; c < CPL; ++c) S[i][c] *= gn[i];
      }
#pragma unroll
      for (int c = 0; c < CPL; ++c) v[c] = vs[tt * COLS + cb + c];
      float u[CPL];
#pragma unroll
      for (int c = 0; c < CPL; ++c) {
        float b0 = 0.f, b1 = 0.f;
        if constexpr (MODE != 2) {
          float a0 = 0.f, a1 = 0.f;
#pragma unroll
          for (int i = 0; i < R; i += 2) {
            a0 = fmaf(S[i][c], k[i], a0);
            a1 = fmaf(S[i + 1][c], k[i + 1], a1);
          }
          u[c] = a0 + a1;
        }
#pragma unroll
        for (int i = 0; i < R; i += 2) {
          b0 = fmaf(S[i][c], q[i], b0);
          b1 = fmaf(S[i + 1][c], q[i + 1], b1);
        }
        part[c][tt] = b0 + b1;
      }
      if constexpr (MODE == 2) {
#pragma unroll
        for (int c = 0; c < CPL; ++c) u[c] = v[c];
      } else {
#pragma unroll
        for (int mask = 8; mask >= 1; mask >>= 1)
#pragma unroll
          for (int c = 0; c < CPL; ++c) u[c] += __shfl_xor_sync(0xffffffffu, u[c], mask);
        // the decayed state answers k with decay * (S^T k); the token writes u along k
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
          u[c] = gate.x * (v[c] - gate.y * u[c]);
          if (l == 0) us[tt * COLS + cb + c] = u[c];             // for the read-out, by lanes of this column only
        }
      }
#pragma unroll
      for (int i = 0; i < R; ++i)
#pragma unroll
        for (int c = 0; c < CPL; ++c) S[i][c] = fmaf(k[i], u[c], MODE == 1 ? S[i][c] : gate.y * S[i][c]);
    };
    if (nt == SEQ_CHUNK) {
#pragma unroll
      for (int tt = 0; tt < SEQ_CHUNK; ++tt) token(tt);
    } else {
#pragma unroll
      for (int tt = 0; tt < SEQ_CHUNK; ++tt) {
        if (tt < nt) token(tt);
        else {
#pragma unroll
          for (int c = 0; c < CPL; ++c) part[c][tt] = 0.f;
        }
      }
    }
    if constexpr (MODE != 2) __syncwarp();
    const int tok = l >> 1;
#pragma unroll
    for (int c = 0; c < CPL; ++c) {
      seq_totals(part[c], l);
      if (!(l & 1) && tok < nt && col + c < P) {
        // the read-out already contains the token's own write: decay * (S^T q) + (k . q) u
        const float4 gate = gates[tok];
        const float u = MODE == 2 ? vs[tok * COLS + cb + c] : us[tok * COLS + cb + c];
        a.o[(size_t)(t0 + tok) * width + (size_t)head * P + col + c] =
            fmaf(gate.z, u, MODE == 1 ? part[c][0] : gate.y * part[c][0]);
      }
    }
    __syncthreads();
  };
  __syncthreads();
  int turn = 0;
  for (int t0 = q0; t0 < q1; t0 += SEQ_CHUNK, turn ^= 1) chunk(t0, turn);
  seq_store_state<NPL, CPL>(st, D, P, col, l, a.vec, S);
}

template <typename AT, int NPL, int WC, int MODE = 0>
static int launch_delta(DeltaArgs a, int S, int T, cudaStream_t stream) {
  constexpr int COLS = SCAN_WARPS * WC;
  a.vec = !(a.P % (WC % 4 == 0 ? 4 : 2)) && !(a.slot_stride % 4) && !((uintptr_t)a.state & 15);
  const dim3 grid((a.P + COLS - 1) / COLS, a.heads, S);
  if (T == S) {
    const size_t one = (size_t)2 * ((MODE == 1 ? 3 : 2) * a.D + COLS + 2) * sizeof(float);
    const cudaError_t e = launch_pdl(delta_scan_kernel<AT, NPL, WC, MODE, 1>, grid, dim3(SCAN_THREADS), one, stream, a);
    return e == cudaSuccess ? FT_OK : (int)e;
  }
  const size_t smem = (size_t)2 * SCAN_CHUNK * ((MODE == 1 ? 3 : 2) * a.D + COLS + 2) * sizeof(float);
  if (smem > 96 * 1024) return FT_ERR_SHAPE;
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(delta_scan_kernel<AT, NPL, WC, MODE, SCAN_CHUNK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaError_t e = launch_pdl(delta_scan_kernel<AT, NPL, WC, MODE, SCAN_CHUNK>, grid, dim3(SCAN_THREADS), smem, stream, a);
  return e == cudaSuccess ? FT_OK : (int)e;
}

template <typename AT, int NPL, int CPL, int MODE>
static int launch_delta_seq(DeltaArgs a, int S, cudaStream_t stream) {
  constexpr size_t smem = 2 * seq_buffer(NPL, CPL, MODE == 1 ? 3 : 2) * sizeof(float);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(delta_seq_kernel<AT, NPL, CPL, MODE>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  a.vec = !(a.P % CPL) && !(a.slot_stride % 4) && !((uintptr_t)a.state & 15) && !((size_t)a.D * a.P % CPL);
  constexpr int COLS = 2 * SEQ_WARPS * CPL;
  const dim3 grid((a.P + COLS - 1) / COLS, a.heads, S);
  const cudaError_t e = launch_pdl(delta_seq_kernel<AT, NPL, CPL, MODE>, grid, dim3(SEQ_THREADS), smem, stream, a);
  return e == cudaSuccess ? FT_OK : (int)e;
}
template <typename AT, int NPL, int MODE>
static int launch_delta_seq(const DeltaArgs& a, int S, cudaStream_t stream) {
  if constexpr (NPL == 8) return launch_delta_seq<AT, NPL, 1, MODE>(a, S, stream);
  else if (sizeof(AT) == 4 || seq_columns(a.P, a.heads, S) == 2) return launch_delta_seq<AT, NPL, 2, MODE>(a, S, stream);
  else if constexpr (sizeof(AT) == 2) return launch_delta_seq<AT, NPL, 4, MODE>(a, S, stream);
  return FT_ERR_DTYPE;
}

template <int MODE>
static int dispatch_delta(DeltaArgs a, int S, int T, int longest, int dtype, cudaStream_t stream) {
  int rc = FT_OK;
  const int D = a.D;
  const bool narrow = narrow_warps(a.P, a.heads, S);
  if (seq_scan(MODE, dtype == FT_DTYPE_F32, a.heads, a.P, D, S, T, longest)) {         // the modes are the first three kinds
    FT_DISPATCH(dtype, AT, {
      if (D <= 32) rc = launch_delta_seq<AT, 1, MODE>(a, S, stream);
      else if (D <= 64) rc = launch_delta_seq<AT, 2, MODE>(a, S, stream);
      else if (D <= 128) rc = launch_delta_seq<AT, 4, MODE>(a, S, stream);
      else rc = launch_delta_seq<AT, 8, MODE>(a, S, stream);
    });
  } else {
    FT_DISPATCH(dtype, AT, {
      if (D <= 32) rc = narrow ? launch_delta<AT, 1, NARROW_WC, MODE>(a, S, T, stream) : launch_delta<AT, 1, 8, MODE>(a, S, T, stream);
      else if (D <= 64) rc = narrow ? launch_delta<AT, 2, NARROW_WC, MODE>(a, S, T, stream) : launch_delta<AT, 2, 8, MODE>(a, S, T, stream);
      else if (D <= 128) rc = narrow ? launch_delta<AT, 4, NARROW_WC, MODE>(a, S, T, stream) : launch_delta<AT, 4, 8, MODE>(a, S, T, stream);
      else rc = narrow ? launch_delta<AT, 8, NARROW_WC, MODE>(a, S, T, stream) : launch_delta<AT, 8, 8, MODE>(a, S, T, stream);
    });
  }
  if (rc != FT_OK) return rc;
  FT_LAUNCH_CHECK();
  return FT_OK;
}

}  // namespace ft
