// Mixers that carry a state of fixed size from token to token: a short causal
// convolution over time and a selective state space with one decay per head
// (Mamba-2's recurrence).  The gated delta rule and retention: delta_scan.cuh; the gated norm
// behind them: gated_norm.cu.
//
//   conv_silu        y[t,c] = silu(b_c + sum_j w[c,j] u[t-(taps-1)+j, c]); the last
//                    taps-1 inputs of a request live in its state slot
//   ssd_scan         S <- exp(-exp(A) dt) S + dt B x^T ; y = S^T C + D x       (S: N x P per head)
//
// A convolution's result depends on its own request alone, however that is cut; what the scans
// hold to, and how a state lies: scans.cuh.
#include "scans.cuh"

namespace ft {

__device__ __forceinline__ float silu_f(float v) { return v / (1.f + expf(-v)); }

// ------------------------------------------------------------ short convolution
struct ConvArgs {
  const void* x;        // [T, ldx]: channel c of token t at x[t * ldx + c]
  void* out;            // [T, ldo]
  const float* w;       // [C, taps]; the last column weighs the current token
  const float* bias;    // [C] or nullptr
  float* state;         // slot s: state + s * slot_stride, [taps - 1][C], oldest input first
  const int* token_seg; // [T]
  const int* seg_slot;  // [S]
  const int* seg_q_start;  // [S + 1]
  long long ldx, ldo, slot_stride;
  int C, taps;
  int act;              // 1: SiLU behind the sum; 0: the sum itself
  int state_ahead;      // the launch right in front does not write the state: it is fetched ahead of the wait
};

constexpr int CONV_MAX_TAPS = 8;     // longer convolutions take the plain loop

// A thread owns one channel (two neighbouring ones where rows allow 4-byte pieces of bfloat16)
// and GROUPS runs of RUN consecutive tokens: while they belong to one segment it keeps the last taps inputs
// in registers and fetches one new input a token, a run ahead; at a segment's first token (and always when
// run is 1) it fetches the whole reach, from earlier rows or from the slot.  The sum runs over
// ascending taps either way.  TAPS: the number of taps where the launch knows it (0: any up to CONV_MAX_TAPS); a
// window of known length is shifted by renaming registers, and several runs share one fetch of the weights
// (conv_groups says when).  bfloat16, four taps, before both and now: 1,024 rows of 512 channels 8.1 -> 6.1 us, 2,048 of
// 2,304 27 -> 16, 4,096 of 6,144 127 -> 73.
template <typename AT, int CPT, int RUN, int TAPS, int GROUPS>
__global__ void __launch_bounds__(128) conv_silu_kernel(ConvArgs a, int T) {
  constexpr int W = TAPS ? TAPS : CONV_MAX_TAPS;
  pdl_wait();
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * CPT;
  if (c >= a.C) return;
  const int K = TAPS ? TAPS - 1 : a.taps - 1;
  const AT* x = (const AT*)a.x;
  float w[CPT][W], win[CPT][W], bias[CPT];
#pragma unroll
  for (int u = 0; u < CPT; ++u) {
    bias[u] = a.bias ? a.bias[c + u] : 0.f;
#pragma unroll
    for (int j = 0; j < W; ++j) w[u][j] = j <= K ? a.w[(size_t)(c + u) * a.taps + j] : 0.f;
  }
  auto fetch = [&](int row, float (&v)[CPT]) {          // CPT inputs of a token's row
    if constexpr (CPT == 2) {
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(x + (size_t)row * a.ldx + c));
      v[0] = f.x;
      v[1] = f.y;
    } else {
      v[0] = to_float(x[(size_t)row * a.ldx + c]);
    }
  };
  int prev_seg = -1;
  const int t_first = blockIdx.x * RUN * GROUPS, t_end = min(T, t_first + RUN * GROUPS);
  // every token's own input and segment of a run first, all loads in flight together, the next run's meanwhile
  float own[RUN][CPT];
  int segs[RUN];
  auto fetch_run = [&](int t0, float (&v)[RUN][CPT], int (&seg)[RUN]) {
#pragma unroll
    for (int i = 0; i < RUN; ++i) {
      if (t0 + i < t_end) {
        fetch(t0 + i, v[i]);
        seg[i] = a.token_seg[t0 + i];
      }
    }
  };
  fetch_run(t_first, own, segs);
  for (int t0 = t_first; t0 < t_end; t0 += RUN) {
    float next[RUN][CPT];
    int next_segs[RUN];
    if constexpr (GROUPS > 1) fetch_run(t0 + RUN, next, next_segs);
#pragma unroll
    for (int i = 0; i < RUN; ++i) {
      const int t = t0 + i;
      if (t >= t_end) break;
      const int seg = segs[i];
      if (seg != prev_seg) {
        const int q0 = a.seg_q_start[seg];
        const int r = t - q0;
        const float* st = a.state + (size_t)a.seg_slot[seg] * a.slot_stride;
#pragma unroll
        for (int j = 0; j < W; ++j) {
          if (j > K) break;
          const int s = r - K + j;
          float v[CPT];
          if (s == r) {
#pragma unroll
            for (int u = 0; u < CPT; ++u) v[u] = own[i][u];
          } else if (s >= 0) fetch(q0 + s, v);
          else {
#pragma unroll
            for (int u = 0; u < CPT; ++u) v[u] = st[(size_t)(K + s) * a.C + c + u];
          }
#pragma unroll
          for (int u = 0; u < CPT; ++u) win[u][j] = v[u];
        }
        prev_seg = seg;
      } else {
#pragma unroll
        for (int u = 0; u < CPT; ++u) {
#pragma unroll
          for (int j = 0; j < W - 1; ++j)
            if (j < K) win[u][j] = win[u][j + 1];
#pragma unroll
          for (int j = 0; j < W; ++j)
            if (j == K) win[u][j] = own[i][u];
        }
      }
      float out[CPT];
#pragma unroll
      for (int u = 0; u < CPT; ++u) {
        float acc = 0.f;
#pragma unroll
        for (int j = 0; j < W; ++j)
          if (j <= K) acc = fmaf(w[u][j], win[u][j], acc);
        out[u] = a.act ? silu_f(acc + bias[u]) : acc + bias[u];
      }
      AT* o = (AT*)a.out + (size_t)t * a.ldo + c;
      if constexpr (CPT == 2) *reinterpret_cast<__nv_bfloat162*>(o) = __floats2bfloat162_rn(out[0], out[1]);
      else o[0] = from_float<AT>(out[0]);
    }
    if constexpr (GROUPS > 1) {
#pragma unroll
      for (int i = 0; i < RUN; ++i) {
        segs[i] = next_segs[i];
#pragma unroll
        for (int u = 0; u < CPT; ++u) own[i][u] = next[i][u];
      }
    }
  }
}

// As many segments as tokens, that is, one token each (decode): a thread owns a segment's channel (or two) with the
// inputs before it in registers, and leaves the last taps - 1 in the slot itself: one launch instead of two, and no
// value read twice.  (One row of 6,144 channels: 2.6 us instead of 2.8 + 2.4.)  It walks whatever tokens the segment has.
template <typename AT, int CPT>
__global__ void __launch_bounds__(128) conv_step_kernel(ConvArgs a) {
  if (!a.state_ahead) pdl_wait();
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * CPT, seg = blockIdx.x;
  const int q0 = a.seg_q_start[seg], q1 = a.seg_q_start[seg + 1], K = a.taps - 1;
  if (c >= a.C || q1 <= q0) {
    if (a.state_ahead) pdl_wait();
    return;
  }
  const AT* x = (const AT*)a.x;
  float* st = a.state + (size_t)a.seg_slot[seg] * a.slot_stride + c;
  float w[CPT][CONV_MAX_TAPS], win[CPT][CONV_MAX_TAPS], bias[CPT];
#pragma unroll
  for (int u = 0; u < CPT; ++u) {
    bias[u] = a.bias ? a.bias[c + u] : 0.f;
#pragma unroll
    for (int j = 0; j < CONV_MAX_TAPS; ++j) {
      w[u][j] = j <= K ? a.w[(size_t)(c + u) * a.taps + j] : 0.f;
      if (j < K) win[u][j] = st[(size_t)j * a.C + u];
    }
  }
  if (a.state_ahead) pdl_wait();
  for (int t = q0; t < q1; ++t) {
    float own[CPT];
    if constexpr (CPT == 2) {
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(x + (size_t)t * a.ldx + c));
      own[0] = f.x;
      own[1] = f.y;
    } else {
      own[0] = to_float(x[(size_t)t * a.ldx + c]);
    }
    float out[CPT];
#pragma unroll
    for (int u = 0; u < CPT; ++u) {
      float acc = 0.f;
#pragma unroll
      for (int j = 0; j < CONV_MAX_TAPS; ++j)
        if (j <= K) acc = fmaf(w[u][j], j == K ? own[u] : win[u][j], acc);
      out[u] = a.act ? silu_f(acc + bias[u]) : acc + bias[u];
#pragma unroll
      for (int j = 0; j < CONV_MAX_TAPS - 1; ++j)
        if (j < K) win[u][j] = j + 1 == K ? own[u] : win[u][j + 1];
    }
    AT* o = (AT*)a.out + (size_t)t * a.ldo + c;
    if constexpr (CPT == 2) *reinterpret_cast<__nv_bfloat162*>(o) = __floats2bfloat162_rn(out[0], out[1]);
    else o[0] = from_float<AT>(out[0]);
  }
#pragma unroll
  for (int u = 0; u < CPT; ++u)
#pragma unroll
    for (int j = 0; j < CONV_MAX_TAPS - 1; ++j)
      if (j < K) st[(size_t)j * a.C + u] = win[u][j];
}

// any number of taps: one channel and one token a thread
template <typename AT>
__global__ void __launch_bounds__(128) conv_silu_long_kernel(ConvArgs a) {
  pdl_wait();
  const int t = blockIdx.x;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= a.C) return;
  const int seg = a.token_seg[t];
  const int q0 = a.seg_q_start[seg];
  const int r = t - q0, K = a.taps - 1;
  const float* st = a.state + (size_t)a.seg_slot[seg] * a.slot_stride;
  const AT* x = (const AT*)a.x;
  float acc = 0.f;
  for (int j = 0; j <= K; ++j) {
    const int s = r - K + j;
    const float v = s >= 0 ? to_float(x[(size_t)(q0 + s) * a.ldx + c]) : st[(size_t)(K + s) * a.C + c];
    acc = fmaf(a.w[(size_t)c * a.taps + j], v, acc);
  }
  if (a.bias) acc += a.bias[c];
  ((AT*)a.out)[(size_t)t * a.ldo + c] = from_float<AT>(a.act ? silu_f(acc) : acc);
}

// After the convolution has read it: the slot keeps the last taps-1 inputs of (what it held ++
// the segment's inputs).  Ascending i reads entries at or above the one it writes.
template <typename AT>
__global__ void __launch_bounds__(128) conv_state_kernel(ConvArgs a) {
  pdl_wait();
  const int seg = blockIdx.x;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  if (c >= a.C) return;
  const int q0 = a.seg_q_start[seg], n = a.seg_q_start[seg + 1] - q0, K = a.taps - 1;
  float* st = a.state + (size_t)a.seg_slot[seg] * a.slot_stride;
  const AT* x = (const AT*)a.x;
  for (int i = 0; i < K; ++i) {
    const int src = n + i;
    st[(size_t)i * a.C + c] = src < K ? st[(size_t)src * a.C + c] : to_float(x[(size_t)(q0 + src - K) * a.ldx + c]);
  }
}

// -------------------------------------------------------- selective state space
struct SsdArgs {
  const void* xbc;      // [T, ld]: x (heads * P) | B (G * N) | C (G * N), after convolution and silu
  const void* dt;       // [T, ld_dt]: the step size's projection, head h at column h
  const float* dt_bias; // [heads]
  const float* A_log;   // [heads]
  const float* D;       // [heads]
  float* state;         // slot s: state + s * slot_stride, [heads][N][P]
  float* y;             // [T, heads * P] float32
  const int* seg_slot;
  const int* seg_q_start;
  long long ld, ld_dt, slot_stride;
  int heads, P, N, G;
  int vec;              // state rows may be read in 16-byte (WC % 4 == 0) or 8-byte pieces
  int state_ahead;      // the launch right in front does not write the state: it is fetched ahead of the wait
};

// NPL: state rows a lane holds (N <= 32 * NPL); WC: state columns a warp owns
// CH: tokens of a chunk; segments of one token each take a chunk of one, whose rows need few registers.
template <typename AT, int NPL, int WC, int CH>
__global__ void __launch_bounds__(SCAN_THREADS) ssd_scan_kernel(SsdArgs a) {
  constexpr int COLS = SCAN_WARPS * WC;
  constexpr int NB = (NPL * 32 + SCAN_THREADS - 1) / SCAN_THREADS;       // B (or C) values a thread stages per token
  constexpr int XR = (CH * COLS + SCAN_THREADS - 1) / SCAN_THREADS;
  extern __shared__ float sm[];
  if (!a.state_ahead) pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int head = blockIdx.y, seg = blockIdx.z;
  const int N = a.N, P = a.P;
  const int g = head / (a.heads / a.G);
  const int inner = a.heads * P;
  const int col0 = blockIdx.x * COLS;
  const int j0 = col0 + warp * WC;
  const int per = CH * (2 * N + COLS + 2);                         // floats of one buffer
  const int q0 = a.seg_q_start[seg], q1 = a.seg_q_start[seg + 1];
  float* st = a.state + (size_t)a.seg_slot[seg] * a.slot_stride + (size_t)head * N * P;
  const float rate = -expf(a.A_log[head]), bias = a.dt_bias[head], skip = a.D[head];
  const AT* xbc = (const AT*)a.xbc;
  const AT* dt = (const AT*)a.dt;

  float S[NPL][WC];
#pragma unroll
  for (int e = 0; e < NPL; ++e) {
    const int n = lane + 32 * e;
    if (n < N) load_cols<WC>(st + (size_t)n * P + j0, S[e], P - j0, a.vec);
    else {
#pragma unroll
      for (int c = 0; c < WC; ++c) S[e][c] = 0.f;
    }
  }
  if (a.state_ahead) pdl_wait();

  AT pb[CH][NB], pc[CH][NB], px[XR], pdt;
  auto fetch = [&](int t0, int nt) {
#pragma unroll
    for (int tt = 0; tt < CH; ++tt) {
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int n = threadIdx.x + SCAN_THREADS * b;
        if (tt < nt && n < N) {
          const AT* row = xbc + (size_t)(t0 + tt) * a.ld + inner + (size_t)g * N + n;
          pb[tt][b] = row[0];
          pc[tt][b] = row[(size_t)a.G * N];
        }
      }
    }
#pragma unroll
    for (int r = 0; r < XR; ++r) {
      const int i = threadIdx.x + SCAN_THREADS * r, tt = i / COLS, c = i % COLS;
      px[r] = (tt < nt && col0 + c < P) ? xbc[(size_t)(t0 + tt) * a.ld + (size_t)head * P + col0 + c] : from_float<AT>(0.f);
    }
    if ((int)threadIdx.x < nt) pdt = dt[(size_t)(t0 + threadIdx.x) * a.ld_dt + head];
  };
  auto put = [&](float* buf, int nt) {
    float* Bs = buf;
    float* Cs = Bs + CH * N;
    float* xs = Cs + CH * N;
    float* dts = xs + CH * COLS;
#pragma unroll
    for (int tt = 0; tt < CH; ++tt) {
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int n = threadIdx.x + SCAN_THREADS * b;
        if (tt < nt && n < N) {
          Bs[tt * N + n] = to_float(pb[tt][b]);
          Cs[tt * N + n] = to_float(pc[tt][b]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < XR; ++r) {
      const int i = threadIdx.x + SCAN_THREADS * r;
      if (i < CH * COLS) xs[i] = to_float(px[r]);
    }
    if ((int)threadIdx.x < nt) {
      const float step = softplus_f(to_float(pdt) + bias);
      dts[threadIdx.x] = step;
      dts[CH + threadIdx.x] = expf(rate * step);
    }
  };

  fetch(q0, min(CH, q1 - q0));
  put(sm, min(CH, q1 - q0));
  __syncthreads();
  int turn = 0;
  for (int t0 = q0; t0 < q1; t0 += CH, turn ^= 1) {
    const int nt = min(CH, q1 - t0);
    const int next = min(CH, q1 - t0 - CH);
    if (next > 0) fetch(t0 + CH, next);
    const float* Bs = sm + turn * per;
    const float* Cs = Bs + CH * N;
    const float* xs = Cs + CH * N;
    const float* dts = xs + CH * COLS;
    auto token = [&](int tt) {
      const float step = dts[tt], decay = dts[CH + tt];
      float Bv[NPL], Cv[NPL];
#pragma unroll
      for (int e = 0; e < NPL; ++e) {
        const int n = lane + 32 * e;
        Bv[e] = n < N ? Bs[tt * N + n] : 0.f;
        Cv[e] = n < N ? Cs[tt * N + n] : 0.f;
      }
      float part[WC], xv[WC];
#pragma unroll
      for (int c = 0; c < WC; ++c) {
        xv[c] = xs[tt * COLS + warp * WC + c];
        const float in = step * xv[c];
        float acc = 0.f;
#pragma unroll
        for (int e = 0; e < NPL; ++e) {
          S[e][c] = fmaf(decay, S[e][c], in * Bv[e]);
          acc = fmaf(S[e][c], Cv[e], acc);
        }
        part[c] = acc;
      }
      warp_sum_multi<WC>(part);
      const int c = lane >> (5 - Log2<WC>::value);
      if ((lane & ((32 / WC) - 1)) == 0 && j0 + c < P) {
        float mine = xv[0];
#pragma unroll
        for (int i = 1; i < WC; ++i) mine = c == i ? xv[i] : mine;
        a.y[(size_t)(t0 + tt) * inner + (size_t)head * P + j0 + c] = part[0] + skip * mine;
      }
    };
    if (nt == CH) {
#pragma unroll
      for (int tt = 0; tt < CH; ++tt) token(tt);
    } else {
      for (int tt = 0; tt < nt; ++tt) token(tt);
    }
    if (next > 0) put(sm + (turn ^ 1) * per, next);
    __syncthreads();
  }
#pragma unroll
  for (int e = 0; e < NPL; ++e) {
    const int n = lane + 32 * e;
    if (n < N) store_cols<WC>(st + (size_t)n * P + j0, S[e], P - j0, a.vec);
  }
}

// The same for the selective state space (ssd_scan_kernel).
template <typename AT, int NPL, int CPL>
__global__ void __launch_bounds__(SEQ_THREADS, NPL < 8 ? 2 : 1) ssd_seq_kernel(SsdArgs a) {
  constexpr int R = 2 * NPL, DP = 32 * NPL, COLS = 2 * SEQ_WARPS * CPL;
  constexpr int PER = seq_buffer(NPL, CPL, 2);
  constexpr int XR = (SEQ_CHUNK * COLS + 32 * SEQ_WARPS - 1) / (32 * SEQ_WARPS);
  extern __shared__ __align__(16) float sm[];
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % SEQ_WARPS, l = lane & 15;
  const bool stages = threadIdx.x >= 32 * SEQ_WARPS;
  const int head = blockIdx.y, seg = blockIdx.z;
  const int N = a.N, P = a.P;
  const int q0 = a.seg_q_start[seg], q1 = a.seg_q_start[seg + 1];
  if (q1 <= q0) return;
  const int g = head / (a.heads / a.G);
  const int inner = a.heads * P;
  const int col0 = blockIdx.x * COLS, cb = (2 * warp + (lane >> 4)) * CPL, col = col0 + cb;
  float* st = a.state + (size_t)a.seg_slot[seg] * a.slot_stride + (size_t)head * N * P;
  const float rate = -expf(a.A_log[head]), bias = a.dt_bias[head], skip = a.D[head];
  const AT* xbc = (const AT*)a.xbc;
  struct Staged {
    AT b[SEQ_PER_WARP][NPL], c[SEQ_PER_WARP][NPL], x[XR], dt[SEQ_PER_WARP];
  } even, odd;
  auto fetch = [&](int t0, Staged& x) {
    const int nt = min(SEQ_CHUNK, q1 - t0);
#pragma unroll
    for (int j = 0; j < SEQ_PER_WARP; ++j) {
      const int tt = warp + SEQ_WARPS * j;
      const size_t t = t0 + tt;
#pragma unroll
      for (int e = 0; e < NPL; ++e) {
        const int n = lane + 32 * e;
        const bool in = tt < nt && n < N;
        const AT* row = xbc + t * a.ld + inner + (size_t)g * N + n;
        x.b[j][e] = in ? row[0] : from_float<AT>(0.f);
        x.c[j][e] = in ? row[(size_t)a.G * N] : from_float<AT>(0.f);
      }
      if (tt < nt) x.dt[j] = ((const AT*)a.dt)[t * a.ld_dt + head];
    }
#pragma unroll
    for (int r = 0; r < XR; ++r) {
      const int i = threadIdx.x % (32 * SEQ_WARPS) + 32 * SEQ_WARPS * r, tt = i / COLS, c = i % COLS;
      x.x[r] = (tt < nt && col0 + c < P) ? xbc[(size_t)(t0 + tt) * a.ld + (size_t)head * P + col0 + c] : from_float<AT>(0.f);
    }
  };
  auto put = [&](float* buf, const Staged& x) {
    float* bs = buf;
    float* cs = bs + SEQ_CHUNK * DP;
    float* xs = cs + SEQ_CHUNK * DP;
    float4* gates = reinterpret_cast<float4*>(xs + SEQ_CHUNK * COLS);      // step, decay
#pragma unroll
    for (int j = 0; j < SEQ_PER_WARP; ++j) {
      const int tt = warp + SEQ_WARPS * j;
#pragma unroll
      for (int e = 0; e < NPL; ++e) {
        const int at = tt * DP + seq_place<NPL>(lane + 32 * e);
        bs[at] = to_float(x.b[j][e]);
        cs[at] = to_float(x.c[j][e]);
      }
    }
    if (lane < SEQ_PER_WARP) {                                   // a lane a token
      AT raw = x.dt[0];
#pragma unroll
      for (int j = 1; j < SEQ_PER_WARP; ++j)
        if (lane == j) raw = x.dt[j];
      const float step = softplus_f(to_float(raw) + bias);
      gates[warp + SEQ_WARPS * lane] = make_float4(step, expf(rate * step), 0.f, 0.f);
    }
#pragma unroll
    for (int r = 0; r < XR; ++r) {
      const int i = threadIdx.x % (32 * SEQ_WARPS) + 32 * SEQ_WARPS * r;
      if (i < SEQ_CHUNK * COLS) xs[i] = to_float(x.x[r]);
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
  seq_load_state<NPL, CPL>(st, N, P, col, l, a.vec, S);
  auto chunk = [&](int t0, int turn) {
    const int nt = min(SEQ_CHUNK, q1 - t0);
    const float* bs = sm + turn * PER;
    const float* cs = bs + SEQ_CHUNK * DP;
    const float* xs = cs + SEQ_CHUNK * DP;
    const float4* gates = reinterpret_cast<const float4*>(xs + SEQ_CHUNK * COLS);
    float part[CPL][SEQ_CHUNK];
    auto token = [&](int tt) {
      float b[R], c[R];
      seq_row<NPL>(bs + tt * DP, l, b);
      seq_row<NPL>(cs + tt * DP, l, c);
      const float4 gate = gates[tt];
#pragma unroll
      for (int j = 0; j < CPL; ++j) {
        const float in = gate.x * xs[tt * COLS + cb + j];
        float p0 = 0.f, p1 = 0.f;
#pragma unroll
        for (int i = 0; i < R; i += 2) {
          S[i][j] = fmaf(gate.y, S[i][j], in * b[i]);
          p0 = fmaf(S[i][j], c[i], p0);
          S[i + 1][j] = fmaf(gate.y, S[i + 1][j], in * b[i + 1]);
          p1 = fmaf(S[i + 1][j], c[i + 1], p1);
        }
        part[j][tt] = p0 + p1;
      }
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
          for (int j = 0; j < CPL; ++j) part[j][tt] = 0.f;
        }
      }
    }
    const int tok = l >> 1;
#pragma unroll
    for (int j = 0; j < CPL; ++j) {
      seq_totals(part[j], l);
      if (!(l & 1) && tok < nt && col + j < P)
        a.y[(size_t)(t0 + tok) * inner + (size_t)head * P + col + j] = part[j][0] + skip * xs[tok * COLS + cb + j];
    }
    __syncthreads();
  };
  __syncthreads();
  int turn = 0;
  for (int t0 = q0; t0 < q1; t0 += SEQ_CHUNK, turn ^= 1) chunk(t0, turn);
  seq_store_state<NPL, CPL>(st, N, P, col, l, a.vec, S);
}

template <typename AT, int NPL, int WC>
static int launch_ssd(SsdArgs a, int S, int T, cudaStream_t stream) {
  constexpr int COLS = SCAN_WARPS * WC;
  const size_t smem = (size_t)2 * SCAN_CHUNK * (2 * a.N + COLS + 2) * sizeof(float);
  if (smem > 48 * 1024) return FT_ERR_SHAPE;
  a.vec = !(a.P % (WC % 4 == 0 ? 4 : 2)) && !(a.slot_stride % 4) && !((uintptr_t)a.state & 15);
  const dim3 grid((a.P + COLS - 1) / COLS, a.heads, S);
  const cudaError_t e =
      T == S ? launch_pdl(ssd_scan_kernel<AT, NPL, WC, 1>, grid, dim3(SCAN_THREADS), smem / SCAN_CHUNK, stream, a)
             : launch_pdl(ssd_scan_kernel<AT, NPL, WC, SCAN_CHUNK>, grid, dim3(SCAN_THREADS), smem, stream, a);
  return e == cudaSuccess ? FT_OK : (int)e;
}

template <typename AT, int NPL, int CPL>
static int launch_ssd_seq(SsdArgs a, int S, cudaStream_t stream) {
  constexpr size_t smem = 2 * seq_buffer(NPL, CPL, 2) * sizeof(float);
  static_assert(smem <= 48 * 1024, "no opt-in needed");
  a.vec = !(a.P % CPL) && !(a.slot_stride % 4) && !((uintptr_t)a.state & 15) && !((size_t)a.N * a.P % CPL);
  constexpr int COLS = 2 * SEQ_WARPS * CPL;
  const dim3 grid((a.P + COLS - 1) / COLS, a.heads, S);
  const cudaError_t e = launch_pdl(ssd_seq_kernel<AT, NPL, CPL>, grid, dim3(SEQ_THREADS), smem, stream, a);
  return e == cudaSuccess ? FT_OK : (int)e;
}
template <typename AT, int NPL>
static int launch_ssd_seq(const SsdArgs& a, int S, cudaStream_t stream) {
  if constexpr (NPL == 8) return launch_ssd_seq<AT, NPL, 1>(a, S, stream);
  else if (sizeof(AT) == 4 || seq_columns(a.P, a.heads, S) == 2) return launch_ssd_seq<AT, NPL, 2>(a, S, stream);
  else if constexpr (sizeof(AT) == 2) return launch_ssd_seq<AT, NPL, 4>(a, S, stream);
  return FT_ERR_DTYPE;
}

// Runs of eight tokens a thread of conv_silu_kernel walks; 0: a thread a token, below 1,024 tokens.  More than one run
// saves fetches of the weights and of the reach, where it leaves blocks enough (1,000 of 128 threads; measured, us with one run and with
// four: 1,024 rows of 512 channels 6.1 and 11.7; two, 4,096 rows of 6,144: 80 and 73) and segments are long (63 single
// tokens beside 961 of 2,304 channels: a window is fetched anew at each, 14 and 26).  Single channels (float32) walk
// four; two channels of other than four taps never gained (4,096 rows of 6,144, three taps: 117 and 129).
static int conv_groups(int C, int T, int S, int taps, bool pairs) {
  if (T < 1024) return 0;
  if (T < 64LL * S) return 1;
  if (pairs) return taps == 4 && (long long)(T / 16) * ((C / 2 + 127) / 128) >= 1000 ? 2 : 1;
  return (long long)(T / 32) * ((C + 127) / 128) >= 1100 ? 4 : 1;
}

}  // namespace ft

using namespace ft;

extern "C" {

int ft_scan_several(int kind, int f32, int heads, int P, int D, int S, int T, int longest) {
  return seq_scan(kind, f32 != 0, heads, P, D, S, T, longest);
}
int ft_conv_groups(int C, int T, int S, int taps, int pairs) { return conv_groups(C, T, S, taps, pairs != 0); }

// Both kernels of the short convolution: outputs first, then the slots' new contents.
int ft_conv_silu(const void* x, long long ldx, void* out, long long ldo, const float* w, const float* bias,
                 float* state, long long slot_stride, const int* token_seg, const int* seg_slot,
                 const int* seg_q_start, int C, int taps, int T, int S, int dtype, int act, int state_ahead,
                 cudaStream_t stream) {
  if (T <= 0 || S <= 0) return FT_OK;
  if (C <= 0 || taps < 1) return FT_ERR_SHAPE;
  ConvArgs a{x, out, w, bias, state, token_seg, seg_slot, seg_q_start, ldx, ldo, slot_stride, C, taps, act, state_ahead};
  const int cb = (C + 127) / 128;
  const bool pairs = dtype == FT_DTYPE_BF16 && !(C & 1) && !(ldx & 1) && !(ldo & 1) && !((uintptr_t)x & 3) &&
                     !((uintptr_t)out & 3);
  if (T == S && taps <= CONV_MAX_TAPS) {
    if (pairs) launch_pdl(conv_step_kernel<__nv_bfloat16, 2>, dim3(S, (C / 2 + 127) / 128), dim3(128), 0, stream, a);
    else FT_DISPATCH(dtype, AT, launch_pdl(conv_step_kernel<AT, 1>, dim3(S, cb), dim3(128), 0, stream, a));
    FT_LAUNCH_CHECK();
    return FT_OK;
  }
  if (taps > CONV_MAX_TAPS) {
    FT_DISPATCH(dtype, AT, launch_pdl(conv_silu_long_kernel<AT>, dim3(T, cb), dim3(128), 0, stream, a));
  } else {
    // many tokens: a thread walks eight of them and more with its inputs in registers; few: a thread a token
    const int groups = conv_groups(C, T, S, taps, pairs);
    const int walked = groups == 0 ? 1 : 8 * groups;
    const dim3 grid((T + walked - 1) / walked, pairs ? (C / 2 + 127) / 128 : cb), block(128);
    using B = __nv_bfloat16;
    if (pairs) {
      if (groups == 0) launch_pdl(conv_silu_kernel<B, 2, 1, 0, 1>, grid, block, 0, stream, a, T);
      else if (taps != 4) launch_pdl(conv_silu_kernel<B, 2, 8, 0, 1>, grid, block, 0, stream, a, T);
      else if (groups == 1) launch_pdl(conv_silu_kernel<B, 2, 8, 4, 1>, grid, block, 0, stream, a, T);
      else launch_pdl(conv_silu_kernel<B, 2, 8, 4, 2>, grid, block, 0, stream, a, T);
    } else if (groups == 0) {
      FT_DISPATCH(dtype, AT, launch_pdl(conv_silu_kernel<AT, 1, 1, 0, 1>, grid, block, 0, stream, a, T));
    } else if (groups == 1) {
      FT_DISPATCH(dtype, AT, launch_pdl(conv_silu_kernel<AT, 1, 8, 0, 1>, grid, block, 0, stream, a, T));
    } else {
      FT_DISPATCH(dtype, AT, launch_pdl(conv_silu_kernel<AT, 1, 8, 0, 4>, grid, block, 0, stream, a, T));
    }
  }
  FT_LAUNCH_CHECK();
  if (taps > 1) {
    FT_DISPATCH(dtype, AT, launch_pdl(conv_state_kernel<AT>, dim3(S, cb), dim3(128), 0, stream, a));
    FT_LAUNCH_CHECK();
  }
  return FT_OK;
}

int ft_ssd_scan(const void* xbc, long long ld, const void* dt, long long ld_dt, const float* dt_bias,
                const float* A_log, const float* D, float* state, long long slot_stride, float* y,
                const int* seg_slot, const int* seg_q_start, int heads, int P, int N, int G, int S,
                int T, int longest, int dtype, int state_ahead, cudaStream_t stream) {
  if (S <= 0) return FT_OK;
  if (heads <= 0 || P <= 0 || N <= 0 || N > 256 || G <= 0 || heads % G) return FT_ERR_SHAPE;
  SsdArgs a{xbc, dt, dt_bias, A_log, D, state, y, seg_slot, seg_q_start, ld, ld_dt, slot_stride, heads, P, N, G, 0, state_ahead};
  int rc = FT_OK;
  const bool narrow = narrow_warps(P, heads, S);
  if (seq_scan(SCAN_SSD, dtype == FT_DTYPE_F32, heads, P, N, S, T, longest)) {
    FT_DISPATCH(dtype, AT, {
      if (N <= 32) rc = launch_ssd_seq<AT, 1>(a, S, stream);
      else if (N <= 64) rc = launch_ssd_seq<AT, 2>(a, S, stream);
      else if (N <= 128) rc = launch_ssd_seq<AT, 4>(a, S, stream);
      else rc = launch_ssd_seq<AT, 8>(a, S, stream);
    });
  } else {
    FT_DISPATCH(dtype, AT, {
      if (N <= 32) rc = narrow ? launch_ssd<AT, 1, NARROW_WC>(a, S, T, stream) : launch_ssd<AT, 1, 8>(a, S, T, stream);
      else if (N <= 64) rc = narrow ? launch_ssd<AT, 2, NARROW_WC>(a, S, T, stream) : launch_ssd<AT, 2, 8>(a, S, T, stream);
      else if (N <= 128) rc = narrow ? launch_ssd<AT, 4, NARROW_WC>(a, S, T, stream) : launch_ssd<AT, 4, 8>(a, S, T, stream);
      else rc = narrow ? launch_ssd<AT, 8, NARROW_WC>(a, S, T, stream) : launch_ssd<AT, 8, 8>(a, S, T, stream);
    });
  }
  if (rc != FT_OK) return rc;
  FT_LAUNCH_CHECK();
  return FT_OK;
}

}  // extern "C"

FT_PACKED(ft_conv_silu)
FT_PACKED(ft_ssd_scan)
