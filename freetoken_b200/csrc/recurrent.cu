// Mixers that carry a state of fixed size from token to token: a short causal
// convolution over time, a selective state space with one decay per head
// (Mamba-2's recurrence) and the gated delta rule (the gated norm behind them: gated_norm.cu).
//
// Everything that enters a recurrence is float32 whatever the activation type:
// step sizes (softplus), decays (exp), gates (sigmoid), unit norms and the state
// itself.  A request's tokens are taken in order; a segment of a step continues
// from the state its request's slot holds and leaves the state there.  A token's
// result depends on its own request alone: on nothing else in the launch, and on
// how the request was cut into steps only through float32 rounding (it is not:
// every token performs the same operations in the same order whatever the cut).
//
//   conv_silu        y[t,c] = silu(b_c + sum_j w[c,j] u[t-(taps-1)+j, c]); the last
//                    taps-1 inputs of a request live in its state slot
//   ssd_scan         S <- exp(-exp(A) dt) S + dt B x^T ; y = S^T C + D x       (S: N x P per head)
//   delta_scan       S <- g S ; u = beta (v - S^T k) ; S <- S + k u^T ; o = S^T q   (S: D x P per head)
//
// State layout per head: [N or D][P] float32, P contiguous.  A warp owns WC
// columns of a head's state and its lanes split the rows, so a column's dot
// products are one warp reduction; a block's four warps share the tokens of a
// chunk, which all threads stage into shared memory together.  Which WC a launch
// takes depends on the step's shape, never on a token's place in it, and the
// operations on a column are the same for every WC.  Launches whose segments have several
// tokens may take kernels with 16 lanes a column that perform the same operations (see
// there, and seq_scan for which).
#include "common.cuh"

namespace ft {

__device__ __forceinline__ float silu_f(float v) { return v / (1.f + expf(-v)); }
__device__ __forceinline__ float softplus_f(float v) { return v > 20.f ? v : log1pf(expf(v)); }
// Sums V values per lane over the warp with V - 1 + log2(32 / V) shuffles: at every step a lane
// hands half of its values to the lane `mask` away and adds what it gets to the half it keeps.
// Afterwards v[0] of lane l is the warp's total of value  l >> (5 - log2 V).
template <int V>
__device__ __forceinline__ void warp_sum_multi(float (&v)[V]) {
  const int lane = threadIdx.x & 31;
  int mask = 16;
#pragma unroll
  for (int w = V / 2; w >= 1; w >>= 1) {
    const bool upper = lane & mask;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const float send = upper ? v[i] : v[i + w];
      const float keep = upper ? v[i + w] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
    }
    mask >>= 1;
  }
  for (; mask >= 1; mask >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], mask);
}
template <int V> struct Log2 { static constexpr int value = 1 + Log2<V / 2>::value; };
template <> struct Log2<1> { static constexpr int value = 0; };

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
  pdl_wait();
  const int c = (blockIdx.y * blockDim.x + threadIdx.x) * CPT, seg = blockIdx.x;
  if (c >= a.C) return;
  const int q0 = a.seg_q_start[seg], q1 = a.seg_q_start[seg + 1], K = a.taps - 1;
  if (q1 <= q0) return;
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
// Both scans share their shape.  A block of four warps owns COLS = 4 * WC columns of one head's
// state in one segment; a warp owns WC of them and its lanes split the rows (NPL rows a lane).
// Tokens come in chunks of SCAN_CHUNK: every thread fetches its share of the NEXT chunk's rows
// into registers before the block works through the current chunk from shared memory, and puts
// them into the other of two buffers afterwards, so that the loads' latency hides under the
// arithmetic and a chunk costs one block-wide barrier.  A full chunk's tokens are unrolled, so
// that the shuffles of one token's read-out overlap the next token's products.
constexpr int SCAN_WARPS = 4;
constexpr int SCAN_THREADS = SCAN_WARPS * 32;
constexpr int SCAN_CHUNK = 8;

// WC consecutive floats of a state row: 16- or 8-byte pieces when `vec` says they are aligned
template <int WC>
__device__ __forceinline__ void load_cols(const float* p, float (&v)[WC], int valid, bool vec) {
  if (WC > 1 && vec && valid >= WC) {
    if constexpr (WC % 4 == 0) {
#pragma unroll
      for (int c = 0; c < WC; c += 4) {
        const float4 f = *reinterpret_cast<const float4*>(p + c);
        v[c] = f.x; v[c + 1] = f.y; v[c + 2] = f.z; v[c + 3] = f.w;
      }
    } else if constexpr (WC % 2 == 0) {
#pragma unroll
      for (int c = 0; c < WC; c += 2) {
        const float2 f = *reinterpret_cast<const float2*>(p + c);
        v[c] = f.x; v[c + 1] = f.y;
      }
    }
    return;
  }
#pragma unroll
  for (int c = 0; c < WC; ++c) v[c] = c < valid ? p[c] : 0.f;
}
template <int WC>
__device__ __forceinline__ void store_cols(float* p, const float (&v)[WC], int valid, bool vec) {
  if (WC > 1 && vec && valid >= WC) {
    if constexpr (WC % 4 == 0) {
#pragma unroll
      for (int c = 0; c < WC; c += 4) *reinterpret_cast<float4*>(p + c) = make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]);
    } else if constexpr (WC % 2 == 0) {
#pragma unroll
      for (int c = 0; c < WC; c += 2) *reinterpret_cast<float2*>(p + c) = make_float2(v[c], v[c + 1]);
    }
    return;
  }
#pragma unroll
  for (int c = 0; c < WC; ++c)
    if (c < valid) p[c] = v[c];
}

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
};

// NPL: state rows a lane holds (N <= 32 * NPL); WC: state columns a warp owns
template <typename AT, int NPL, int WC>
__global__ void __launch_bounds__(SCAN_THREADS) ssd_scan_kernel(SsdArgs a) {
  constexpr int COLS = SCAN_WARPS * WC;
  constexpr int NB = (NPL * 32 + SCAN_THREADS - 1) / SCAN_THREADS;       // B (or C) values a thread stages per token
  constexpr int XR = (SCAN_CHUNK * COLS + SCAN_THREADS - 1) / SCAN_THREADS;
  extern __shared__ float sm[];
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int head = blockIdx.y, seg = blockIdx.z;
  const int N = a.N, P = a.P;
  const int g = head / (a.heads / a.G);
  const int inner = a.heads * P;
  const int col0 = blockIdx.x * COLS;
  const int j0 = col0 + warp * WC;
  const int per = SCAN_CHUNK * (2 * N + COLS + 2);                         // floats of one buffer
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

  AT pb[SCAN_CHUNK][NB], pc[SCAN_CHUNK][NB], px[XR], pdt;
  auto fetch = [&](int t0, int nt) {
#pragma unroll
    for (int tt = 0; tt < SCAN_CHUNK; ++tt) {
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
    float* Cs = Bs + SCAN_CHUNK * N;
    float* xs = Cs + SCAN_CHUNK * N;
    float* dts = xs + SCAN_CHUNK * COLS;
#pragma unroll
    for (int tt = 0; tt < SCAN_CHUNK; ++tt) {
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
      if (i < SCAN_CHUNK * COLS) xs[i] = to_float(px[r]);
    }
    if ((int)threadIdx.x < nt) {
      const float step = softplus_f(to_float(pdt) + bias);
      dts[threadIdx.x] = step;
      dts[SCAN_CHUNK + threadIdx.x] = expf(rate * step);
    }
  };

  fetch(q0, min(SCAN_CHUNK, q1 - q0));
  put(sm, min(SCAN_CHUNK, q1 - q0));
  __syncthreads();
  int turn = 0;
  for (int t0 = q0; t0 < q1; t0 += SCAN_CHUNK, turn ^= 1) {
    const int nt = min(SCAN_CHUNK, q1 - t0);
    const int next = min(SCAN_CHUNK, q1 - t0 - SCAN_CHUNK);
    if (next > 0) fetch(t0 + SCAN_CHUNK, next);
    const float* Bs = sm + turn * per;
    const float* Cs = Bs + SCAN_CHUNK * N;
    const float* xs = Cs + SCAN_CHUNK * N;
    const float* dts = xs + SCAN_CHUNK * COLS;
    auto token = [&](int tt) {
      const float step = dts[tt], decay = dts[SCAN_CHUNK + tt];
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
    if (nt == SCAN_CHUNK) {
#pragma unroll
      for (int tt = 0; tt < SCAN_CHUNK; ++tt) token(tt);
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

// ------------------------------------------------------------- gated delta rule
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
};

// MODE 0: the gated delta rule with one decay per head.
// MODE 1: the same rule with a decay per key channel: row n of a head's state is multiplied by
//         g_n = exp(-exp(A_log_h) softplus(a_n + dt_bias[h * D + n])) before the token reads and writes.
// MODE 2: retention: S <- c_h S + k v^T, o = S^T q with a constant c_h per head (dt_bias[h]), no write
//         strength and no unit norms; q and k have the first rot_dims dimensions of each head turned
//         by the token's position (dimension i with i + rot_dims / 2) in shared memory, in float32;
//         k is multiplied by q_scale after the rotation.
template <typename AT, int NPL, int WC, int MODE>
__global__ void __launch_bounds__(SCAN_THREADS) delta_scan_kernel(DeltaArgs a) {
  constexpr int COLS = SCAN_WARPS * WC;
  constexpr int NB = (NPL * 32 + SCAN_THREADS - 1) / SCAN_THREADS;
  constexpr int XR = (SCAN_CHUNK * COLS + SCAN_THREADS - 1) / SCAN_THREADS;
  extern __shared__ float sm[];
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int head = blockIdx.y, seg = blockIdx.z;
  const int D = a.D, P = a.P;
  const int g = head / (a.heads / a.G);
  const int col0 = blockIdx.x * COLS;
  const int j0 = col0 + warp * WC;
  const int width = a.heads * P;
  const int per = SCAN_CHUNK * ((MODE == 1 ? 3 : 2) * D + COLS + 2);
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

  AT pq[SCAN_CHUNK][NB], pk[SCAN_CHUNK][NB], pv[XR], pbeta, pdecay;
  float pg[MODE == 1 ? SCAN_CHUNK : 1][NB];                   // MODE 1: the channels' decay projections
  float pcos[MODE == 2 ? NPL : 1], psin[MODE == 2 ? NPL : 1]; // MODE 2: pair (tt, i) = threadIdx.x + 128 r
  auto fetch = [&](int t0, int nt) {
#pragma unroll
    for (int tt = 0; tt < SCAN_CHUNK; ++tt) {
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
    float* ks = qs + SCAN_CHUNK * D;
    float* vs = ks + SCAN_CHUNK * D;
    float* gates = vs + SCAN_CHUNK * COLS;
#pragma unroll
    for (int tt = 0; tt < SCAN_CHUNK; ++tt) {
#pragma unroll
      for (int b = 0; b < NB; ++b) {
        const int n = threadIdx.x + SCAN_THREADS * b;
        if (tt < nt && n < D) {
          qs[tt * D + n] = to_float(pq[tt][b]);
          ks[tt * D + n] = to_float(pk[tt][b]);
          if constexpr (MODE == 1)
            gates[2 * SCAN_CHUNK + tt * D + n] = expf(rate * softplus_f(pg[tt][b] + ch_bias[b]));
        }
      }
    }
#pragma unroll
    for (int r = 0; r < XR; ++r) {
      const int i = threadIdx.x + SCAN_THREADS * r;
      if (i < SCAN_CHUNK * COLS) vs[i] = to_float(pv[r]);
    }
    if ((int)threadIdx.x < nt) {
      if constexpr (MODE == 2) {
        gates[threadIdx.x] = 1.f;
        gates[SCAN_CHUNK + threadIdx.x] = bias;
      } else {
        gates[threadIdx.x] = 1.f / (1.f + expf(-to_float(pbeta)));
        gates[SCAN_CHUNK + threadIdx.x] = MODE == 1 ? 1.f : expf(rate * softplus_f(to_float(pdecay) + bias));
      }
    }
  };
  // MODE 2: turn the staged q and k rows of a chunk; a thread owns whole pairs
  auto turn_rows = [&](float* buf, int nt) {
    if constexpr (MODE == 2) {
      float* qs = buf;
      float* ks = qs + SCAN_CHUNK * D;
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

  fetch(q0, min(SCAN_CHUNK, q1 - q0));
  put(sm, min(SCAN_CHUNK, q1 - q0));
  if constexpr (MODE == 2) {
    __syncthreads();
    turn_rows(sm, min(SCAN_CHUNK, q1 - q0));
  }
  __syncthreads();
  int turn = 0;
  for (int t0 = q0; t0 < q1; t0 += SCAN_CHUNK, turn ^= 1) {
    const int nt = min(SCAN_CHUNK, q1 - t0);
    const int next = min(SCAN_CHUNK, q1 - t0 - SCAN_CHUNK);
    if (next > 0) fetch(t0 + SCAN_CHUNK, next);
    const float* qs = sm + turn * per;
    const float* ks = qs + SCAN_CHUNK * D;
    const float* vs = ks + SCAN_CHUNK * D;
    const float* gates = vs + SCAN_CHUNK * COLS;
    auto token = [&](int tt) {
      const float beta = gates[tt], decay = gates[SCAN_CHUNK + tt];
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
          const float gn = n < D ? gates[2 * SCAN_CHUNK + tt * D + n] : 1.f;
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
    if (nt == SCAN_CHUNK) {
#pragma unroll
      for (int tt = 0; tt < SCAN_CHUNK; ++tt) token(tt);
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

// ------------------------------------------------- segments of several tokens
// A prompt portion's tokens are a chain, and the kernels above spend a microsecond and more on four of them: 32
// lanes a column, five shuffle stages for the unit vectors, five for the column sums, a broadcast.  Here a column
// belongs to 16 lanes; lane l keeps rows l + 32 e and l + 16 + 32 e of CPL columns, sums them in two chains (what
// lanes l and l + 16 sum above) and adds the two, so that four shuffle stages remain and every sum has the bits of
// the kernels above: which of the two a launch takes does not show in the results.  What does not wait for the
// state (unit vectors, gates, rotations, k . q) is done while a chunk is staged, a warp a token; what nothing waits
// for (the read-outs) is added over the lanes once a chunk, for its eight tokens together.  q and k rows lie in
// shared memory in the lanes' order, so that a lane reads its rows in 16-byte pieces.  Four warps work and four stage (the staging's chain of
// sums, roots and exponentials is as long as eight tokens' work), with two more chunks on their way in registers.
// A chain of eight tokens is bound by its own latency, many segments by issue slots.  Measured, before and now
// (us): one segment of 2,048 tokens, 16 heads of 128 x 128: delta rule 1,037 -> 347, with a decay per channel 1,469
// -> 575, retention 904 -> 338; 32 heads of 64 x 128 of the state space 579 -> 203.  Four segments of 640 .. 1,335
// tokens, 32 heads (64): 1,364 -> 750, 1,665 -> 1,049, 1,257 -> 598, 709 -> 427.
constexpr int SEQ_WARPS = 4;
constexpr int SEQ_THREADS = 64 * SEQ_WARPS;           // as many warps stage as work
constexpr int SEQ_CHUNK = 8;
constexpr int SEQ_PER_WARP = SEQ_CHUNK / SEQ_WARPS;    // tokens a staging warp takes of a chunk

// place of row n in a staged row: lane n & 15 holds its rows one behind the other, in pieces of four (two)
template <int NPL>
__device__ __forceinline__ int seq_place(int n) {
  const int l = n & 15, i = ((n >> 4) & 1) + 2 * (n >> 5);
  return NPL == 1 ? 2 * l + i : (i >> 2) * 64 + 4 * l + (i & 3);
}
template <int NPL>
__device__ __forceinline__ void seq_row(const float* row, int l, float (&v)[2 * NPL]) {
  if constexpr (NPL == 1) {
    const float2 f = *reinterpret_cast<const float2*>(row + 2 * l);
    v[0] = f.x; v[1] = f.y;
  } else {
#pragma unroll
    for (int i = 0; i < 2 * NPL; i += 4) {
      const float4 f = *reinterpret_cast<const float4*>(row + 16 * i + 4 * l);
      v[i] = f.x; v[i + 1] = f.y; v[i + 2] = f.z; v[i + 3] = f.w;
    }
  }
}
// part[t] of the 16 lanes of a column summed: lane l ends with token l >> 1
__device__ __forceinline__ void seq_totals(float (&part)[SEQ_CHUNK], int l) {
  int mask = 8;
#pragma unroll
  for (int w = SEQ_CHUNK / 2; w >= 1; w >>= 1) {
    const bool upper = l & mask;
#pragma unroll
    for (int i = 0; i < w; ++i) {
      const float send = upper ? part[i] : part[i + w];
      const float keep = upper ? part[i + w] : part[i];
      part[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
    }
    mask >>= 1;
  }
  part[0] += __shfl_xor_sync(0xffffffffu, part[0], 1);
}
// the columns of row n that a lane owns
template <int NPL, int CPL>
__device__ __forceinline__ void seq_load_state(const float* st, int rows, int P, int col, int l, bool vec,
                                               float (&S)[2 * NPL][CPL]) {
#pragma unroll
  for (int i = 0; i < 2 * NPL; ++i) {
    const int n = l + 16 * i;
    if (n < rows) load_cols<CPL>(st + (size_t)n * P + col, S[i], P - col, vec);
    else {
#pragma unroll
      for (int c = 0; c < CPL; ++c) S[i][c] = 0.f;
    }
  }
}
template <int NPL, int CPL>
__device__ __forceinline__ void seq_store_state(float* st, int rows, int P, int col, int l, bool vec,
                                                const float (&S)[2 * NPL][CPL]) {
#pragma unroll
  for (int i = 0; i < 2 * NPL; ++i) {
    const int n = l + 16 * i;
    if (n < rows) store_cols<CPL>(st + (size_t)n * P + col, S[i], P - col, vec);
  }
}

constexpr int seq_buffer(int npl, int cpl, int rows) {           // floats of one buffer: rows of 32 npl, columns, gates
  return SEQ_CHUNK * (rows * 32 * npl + 2 * SEQ_WARPS * cpl + 4);
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

// Few columns in all (single tokens of a few requests, short portions) leave most SMs without a block when a warp owns
// 8 of them: then a warp owns 2 and four times as many blocks share the work.
#ifndef NARROW_WC
#define NARROW_WC 2
#endif
static bool narrow_warps(int P, int heads, int S) {
  int sms = 148, dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return (long long)((P + 31) / 32) * heads * S < 2LL * sms;
}

template <typename AT, int NPL, int WC>
static int launch_ssd(SsdArgs a, int S, cudaStream_t stream) {
  constexpr int COLS = SCAN_WARPS * WC;
  const size_t smem = (size_t)2 * SCAN_CHUNK * (2 * a.N + COLS + 2) * sizeof(float);
  if (smem > 48 * 1024) return FT_ERR_SHAPE;
  a.vec = !(a.P % (WC % 4 == 0 ? 4 : 2)) && !(a.slot_stride % 4) && !((uintptr_t)a.state & 15);
  const dim3 grid((a.P + COLS - 1) / COLS, a.heads, S);
  cudaError_t e = launch_pdl(ssd_scan_kernel<AT, NPL, WC>, grid, dim3(SCAN_THREADS), smem, stream, a);
  return e == cudaSuccess ? FT_OK : (int)e;
}

template <typename AT, int NPL, int WC, int MODE = 0>
static int launch_delta(DeltaArgs a, int S, cudaStream_t stream) {
  constexpr int COLS = SCAN_WARPS * WC;
  const size_t smem = (size_t)2 * SCAN_CHUNK * ((MODE == 1 ? 3 : 2) * a.D + COLS + 2) * sizeof(float);
  if (smem > 96 * 1024) return FT_ERR_SHAPE;
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(delta_scan_kernel<AT, NPL, WC, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  a.vec = !(a.P % (WC % 4 == 0 ? 4 : 2)) && !(a.slot_stride % 4) && !((uintptr_t)a.state & 15);
  const dim3 grid((a.P + COLS - 1) / COLS, a.heads, S);
  cudaError_t e = launch_pdl(delta_scan_kernel<AT, NPL, WC, MODE>, grid, dim3(SCAN_THREADS), smem, stream, a);
  return e == cudaSuccess ? FT_OK : (int)e;
}

// Columns a lane of the kernels for several tokens a segment.  Four need fewer shared loads and less staging a
// column, two leave twice as many blocks: measured, two win while the columns of a launch (heads, segments) fill
// the chip once (4,096: delta 499 against 594 us for 2,048 tokens), four from there on (16,384: 911 against 750).
static int seq_columns(int P, int heads, int S) { return (long long)P * heads * S <= 5000 ? 2 : 4; }

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

// Which kernels take T tokens in S segments: those with 16 lanes a column (true) or those with 32.  The former take a third
// of the time a token of a chain and read and write states in narrower pieces, so that they pay with the tokens a state
// stays in registers for, and with a long chain's share of the launch; `longest`: tokens of the longest segment (0: not
// known, the mean).  All lines from both kernels' times over S = 1 .. 64 segments of 2 .. 256 tokens, even ones and a
// long one beside single tokens, heads of 64, 128 and 256 (bfloat16, 16 heads of 128, delta rule, us with 32 and 16
// lanes: 32 segments of 2 tokens 29 and 39, of 16 91 and 73; 31 single tokens beside 16 tokens 36 and 42, beside 128 105
// and 71).  Up to 8,192 columns every block finds a place at once: from the first tokens on.  More: where the long
// segment's chain outlasts the other segments' states, or all segments have several tokens.  Float32 launches take
// two columns a lane and pay later, states of more than 128 rows one: there only long segments that nothing else
// outweighs.
enum ScanKind { SCAN_DELTA, SCAN_CHANNEL, SCAN_RETENTION, SCAN_SSD };
static bool seq_scan(int kind, bool f32, int heads, int P, int D, int S, int T, int longest) {
  if (T <= S) return false;
  const long long head_columns = (long long)heads * P, columns = head_columns * S;
  const long long L = longest > 0 ? longest : (T + S - 1) / S;
  const bool light = kind == SCAN_DELTA || kind == SCAN_SSD;       // a scalar decay a head, nothing turned
  if (D > 128) {
    const bool alone = T <= 2 * L;
    if (columns > 8192) return alone && L * (kind == SCAN_DELTA ? 300 : kind == SCAN_SSD ? 128 : 64) >= columns;
    return light && L >= (kind == SCAN_SSD && columns > 4096 ? 128 : 32);
  }
  if (columns <= 8192) return L >= 4 || (columns > 4096 && (light || !f32));
  constexpr int chain[2][4] = {{1600, 1600, 1600, 1600}, {1024, 700, 800, 512}};       // columns a chain's token stands for
  constexpr int tokens[2][4] = {{8, 8, 8, 12}, {28, 42, 16, 90}};                       // mean tokens more than one
  // float32 work gains little a token: there the others' tokens count against the chain
  const long long beside = f32 ? head_columns * (S + T - L) / 2 : columns;
  return L * chain[f32][kind] >= beside || T - S >= (long long)tokens[f32][kind] * S;
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
      if (D <= 32) rc = narrow ? launch_delta<AT, 1, NARROW_WC, MODE>(a, S, stream) : launch_delta<AT, 1, 8, MODE>(a, S, stream);
      else if (D <= 64) rc = narrow ? launch_delta<AT, 2, NARROW_WC, MODE>(a, S, stream) : launch_delta<AT, 2, 8, MODE>(a, S, stream);
      else if (D <= 128) rc = narrow ? launch_delta<AT, 4, NARROW_WC, MODE>(a, S, stream) : launch_delta<AT, 4, 8, MODE>(a, S, stream);
      else rc = narrow ? launch_delta<AT, 8, NARROW_WC, MODE>(a, S, stream) : launch_delta<AT, 8, 8, MODE>(a, S, stream);
    });
  }
  if (rc != FT_OK) return rc;
  FT_LAUNCH_CHECK();
  return FT_OK;
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
                 const int* seg_q_start, int C, int taps, int T, int S, int dtype, int act, cudaStream_t stream) {
  if (T <= 0 || S <= 0) return FT_OK;
  if (C <= 0 || taps < 1) return FT_ERR_SHAPE;
  ConvArgs a{x, out, w, bias, state, token_seg, seg_slot, seg_q_start, ldx, ldo, slot_stride, C, taps, act};
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
                int T, int longest, int dtype, cudaStream_t stream) {
  if (S <= 0) return FT_OK;
  if (heads <= 0 || P <= 0 || N <= 0 || N > 256 || G <= 0 || heads % G) return FT_ERR_SHAPE;
  SsdArgs a{xbc, dt, dt_bias, A_log, D, state, y, seg_slot, seg_q_start, ld, ld_dt, slot_stride, heads, P, N, G, 0};
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
      if (N <= 32) rc = narrow ? launch_ssd<AT, 1, NARROW_WC>(a, S, stream) : launch_ssd<AT, 1, 8>(a, S, stream);
      else if (N <= 64) rc = narrow ? launch_ssd<AT, 2, NARROW_WC>(a, S, stream) : launch_ssd<AT, 2, 8>(a, S, stream);
      else if (N <= 128) rc = narrow ? launch_ssd<AT, 4, NARROW_WC>(a, S, stream) : launch_ssd<AT, 4, 8>(a, S, stream);
      else rc = narrow ? launch_ssd<AT, 8, NARROW_WC>(a, S, stream) : launch_ssd<AT, 8, 8>(a, S, stream);
    });
  }
  if (rc != FT_OK) return rc;
  FT_LAUNCH_CHECK();
  return FT_OK;
}

int ft_delta_scan(const void* qkv, long long ld, const void* beta, const void* decay, long long ld_gate,
                  const float* dt_bias, const float* A_log, float* state, long long slot_stride, float* o,
                  const int* seg_slot, const int* seg_q_start, int heads, int P, int D, int G, float unit_eps,
                  float q_scale, int S, int T, int longest, int dtype, cudaStream_t stream) {
  if (S <= 0) return FT_OK;
  if (heads <= 0 || P <= 0 || D <= 0 || D > 256 || G <= 0 || heads % G) return FT_ERR_SHAPE;
  DeltaArgs a{qkv, beta, decay, dt_bias, A_log, state, o, seg_slot, seg_q_start, ld, ld_gate, slot_stride,
              heads, P, D, G, unit_eps, q_scale, 0, nullptr, 0, nullptr, nullptr, 0};
  return dispatch_delta<0>(a, S, T, longest, dtype, stream);
}

// The delta rule with a decay per key channel: `decay` is float32 [T, ld_decay] (channel n of head
// h at column h * D + n), dt_bias [heads * D].
int ft_channel_delta_scan(const void* qkv, long long ld, const void* beta, long long ld_gate, const float* decay,
                          long long ld_decay, const float* dt_bias, const float* A_log, float* state,
                          long long slot_stride, float* o, const int* seg_slot, const int* seg_q_start, int heads,
                          int P, int D, int G, float unit_eps, float q_scale, int S, int T, int longest, int dtype,
                          cudaStream_t stream) {
  if (S <= 0) return FT_OK;
  if (heads <= 0 || P <= 0 || D <= 0 || D > 256 || G <= 0 || heads % G) return FT_ERR_SHAPE;
  DeltaArgs a{qkv, beta, nullptr, dt_bias, A_log, state, o, seg_slot, seg_q_start, ld, ld_gate, slot_stride,
              heads, P, D, G, unit_eps, q_scale, 0, decay, ld_decay, nullptr, nullptr, 0};
  return dispatch_delta<1>(a, S, T, longest, dtype, stream);
}

// Retention: rows of `qkv` are q (heads * D) | k (heads * D) | v (heads * P); `decay` [heads] float32 holds
// each head's constant factor; cos_sin [positions, rot_dims] (rot_dims 0: nothing turns).
int ft_retention_scan(const void* qkv, long long ld, const float* decay, const float* cos_sin, int rot_dims,
                      const int* seg_pos0, float* state, long long slot_stride, float* o, const int* seg_slot,
                      const int* seg_q_start, int heads, int P, int D, float k_scale, int S, int T, int longest, int dtype,
                      cudaStream_t stream) {
  if (S <= 0) return FT_OK;
  if (heads <= 0 || P <= 0 || D <= 0 || D > 256 || rot_dims < 0 || (rot_dims & 1) || rot_dims > D)
    return FT_ERR_SHAPE;
  DeltaArgs a{qkv, nullptr, nullptr, decay, nullptr, state, o, seg_slot, seg_q_start, ld, 0, slot_stride,
              heads, P, D, heads, 0.f, k_scale, 0, nullptr, 0, cos_sin, seg_pos0, cos_sin ? rot_dims : 0};
  return dispatch_delta<2>(a, S, T, longest, dtype, stream);
}

}  // extern "C"
