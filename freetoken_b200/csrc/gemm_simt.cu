// C = A * W^T on CUDA cores in float32, dense or grouped by expert.
//
// This is the true 32-bit matrix path (no tensor cores, no reduced-precision
// mode) and the fallback for sizes the tensor-core kernels refuse.  Every
// output element is one thread's sum over k = 0..K-1 in ascending order, so a
// row's result does not depend on how many rows the launch holds, on the tile
// shape chosen, or on which expert group the row fell into.
//
// Four kernels share that arithmetic: gemm_stream_kernel (few rows: the weights are
// streamed once), gemm_tile_kernel (many rows: register tiles), gemm_dense_kernel (between
// the two) and gemm_rows_kernel (any size and alignment).  gemm_route() says which takes what.
//
// Grouped use (routed experts; reference python/freetoken/moe/fused.py:267-337,
// python/freetoken/kernel/triton/fused_moe.py:156-302): rows are sorted by
// expert, group_offsets[g]..group_offsets[g+1] are expert g's rows, W holds one
// [N,K] matrix per expert.  a_rows / c_rows redirect the input and output rows
// (token of a sorted route; route of a sorted row); row_scale multiplies the
// float32 accumulator before rounding (route weight, fused_moe.py:292-296).
// The SwiGLU epilogue reads W as [gate rows 0..N-1 ; up rows N..2N-1] and
// stores act(gate)*up (python/freetoken/kernel/triton/activation.py:96-107).
#include "common.cuh"
#include "mma_utils.cuh"

namespace ft {

struct GemmArgs {
  const void* A;
  const void* W;
  void* C;
  const int* group_offsets;  // [G+1] or nullptr (one group of M rows)
  const int* a_rows;         // [M] or nullptr
  const int* c_rows;         // [M] or nullptr
  const float* row_scale;    // indexed by output row, or nullptr
  long long lda, ldc, w_group_stride;
  int M, N, K, G;
  int act;  // 0 silu(g)*u, 1 swigluoai
  float act_alpha, act_limit;
  // batched use (one product per head of a mixer): blockIdx.z picks the batch, whose
  // A, W and C start this many elements further on
  long long a_batch_stride = 0, w_batch_stride = 0, c_batch_stride = 0;
  int batch = 1;
  bool ahead = false;        // promised_ahead
};

__device__ __forceinline__ float glu_act(float g, float u, int act, float alpha, float limit) {
  if (act == 0) return (g / (1.f + expf(-g))) * u;
  // swigluoai: min(g,L) * sigmoid(alpha*min(g,L)) * (clamp(u,-L,L) + 1)
  g = fminf(g, limit);
  u = fminf(fmaxf(u, -limit), limit);
  return (g / (1.f + expf(-alpha * g))) * (u + 1.f);
}

// Warp 0 writes {group, first row, rows} of row tile blockIdx.x (rows 0: nothing to do): the groups' tile
// counts are summed 32 groups at a time.
template <int BM>
__device__ __forceinline__ void find_tile(const GemmArgs& a, int* info) {
  if (threadIdx.x >= 32) return;
  if (!a.group_offsets) {
    if (threadIdx.x == 0) {
      info[0] = 0;
      info[1] = blockIdx.x * BM;
      info[2] = min(BM, a.M - (int)blockIdx.x * BM);
    }
    return;
  }
  const int tile = blockIdx.x, lane = threadIdx.x;
  int before = 0;
  for (int g0 = 0; g0 < a.G; g0 += 32) {
    const int g = g0 + lane;
    const int begin = g < a.G ? a.group_offsets[g] : 0, end = g < a.G ? a.group_offsets[g + 1] : 0;
    const int nt = (end - begin + BM - 1) / BM;
    int upto = nt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += v;
    }
    const int first = before + upto - nt;
    const bool mine = tile >= first && tile < first + nt;
    if (mine) {
      info[0] = g;
      info[1] = begin + (tile - first) * BM;
      info[2] = min(BM, end - info[1]);
    }
    if (__any_sync(0xffffffffu, mine)) return;
    before += __shfl_sync(0xffffffffu, upto, 31);
  }
  if (lane == 0) info[2] = 0;
}

constexpr int BN = 64;
constexpr int BK = 32;

// Any K, any alignment.
template <typename AT, typename WT, typename OT, int BM, bool GLU>
__global__ void __launch_bounds__(256) gemm_rows_kernel(GemmArgs a) {
  constexpr int TM = BM / 16, TN = BN / 16;
  __shared__ float As[BM][BK + 1];
  __shared__ float Ws[BN][BK + 1];
  __shared__ float Us[GLU ? BN : 1][BK + 1];
  __shared__ int tile_info[3];  // group, first row, rows
  pdl_wait_only();
  find_tile<BM>(a, tile_info);
  __syncthreads();
  const int group = tile_info[0], row0 = tile_info[1], rows = tile_info[2];
  if (rows <= 0) return;
  const int n0 = blockIdx.y * BN;
  const AT* A = (const AT*)a.A + (size_t)blockIdx.z * a.a_batch_stride;
  const WT* W = (const WT*)a.W + (size_t)group * a.w_group_stride + (size_t)blockIdx.z * a.w_batch_stride;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;

  float acc[TM][TN], acu[GLU ? TM : 1][GLU ? TN : 1];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      acc[i][j] = 0.f;
      if (GLU) acu[i][j] = 0.f;
    }

  for (int k0 = 0; k0 < a.K; k0 += BK) {
    for (int idx = threadIdx.x; idx < BM * BK; idx += 256) {
      const int r = idx / BK, kk = idx % BK;
      float v = 0.f;
      if (r < rows && k0 + kk < a.K) {
        const int src = a.a_rows ? a.a_rows[row0 + r] : row0 + r;
        v = to_float(A[(size_t)src * a.lda + k0 + kk]);
      }
      As[r][kk] = v;
    }
    for (int idx = threadIdx.x; idx < BN * BK; idx += 256) {
      const int n = idx / BK, kk = idx % BK;
      float v = 0.f, u = 0.f;
      if (n0 + n < a.N && k0 + kk < a.K) {
        v = to_float(W[(size_t)(n0 + n) * a.K + k0 + kk]);
        if (GLU) u = to_float(W[(size_t)(a.N + n0 + n) * a.K + k0 + kk]);
      }
      Ws[n][kk] = v;
      if (GLU) Us[n][kk] = u;
    }
    __syncthreads();
#pragma unroll 8
    for (int kk = 0; kk < BK; ++kk) {
      float av[TM], wv[TN], uv[GLU ? TN : 1];
#pragma unroll
      for (int i = 0; i < TM; ++i) av[i] = As[ty + 16 * i][kk];
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        wv[j] = Ws[tx + 16 * j][kk];
        if (GLU) uv[j] = Us[tx + 16 * j][kk];
      }
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
          if (GLU) acu[i][j] = fmaf(av[i], uv[j], acu[i][j]);
        }
    }
    __syncthreads();
  }

  OT* C = (OT*)a.C + (size_t)blockIdx.z * a.c_batch_stride;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int r = ty + 16 * i;
    if (r >= rows) continue;
    const int crow = a.c_rows ? a.c_rows[row0 + r] : row0 + r;
    const float scale = a.row_scale ? a.row_scale[crow] : 1.f;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + 16 * j;
      if (n >= a.N) continue;
      float v = acc[i][j];
      if (GLU) v = glu_act(v, acu[i][j], a.act, a.act_alpha, a.act_limit);
      if (a.row_scale) v *= scale;
      C[(size_t)crow * a.ldc + n] = from_float<OT>(v);
    }
  }
}

__device__ __forceinline__ void load8(const float* p, float (&v)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  const float4 b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}
// Two fused multiply-adds in one instruction; each half rounds like fmaf.
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long x, unsigned long long y) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(y));
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}

template <typename OT, bool GLU>
__device__ __forceinline__ void store_out(const GemmArgs& a, OT* C, int crow, int n, float v, float up) {
  if (GLU) v = glu_act(v, up, a.act, a.act_alpha, a.act_limit);
  if (a.row_scale) v *= a.row_scale[crow];
  C[(size_t)crow * a.ldc + n] = from_float<OT>(v);
}

// Few rows: the launch is bound by the weights it streams and, below that, by the one chain of K fused
// multiply-adds an output is (4 cycles each: 4.3 us for K = 2048).  A lane owns a column, a warp R of the
// block's MR rows; weights and rows come through STREAM_STAGES cp.async stages of STREAM_K values of k, so
// that a block keeps three stages in flight and no thread's load waits for its arithmetic.  (The plain kernel
// loads a 32-wide k tile, waits, multiplies and waits again: 53 products of two rows, K = 2048, N = 2048 .. 32768, took
// 13,350 us and take 1,014.)  Weight rows are padded by 16 bytes: a quarter warp's 16-byte reads touch all banks.
constexpr int STREAM_K = 128;
constexpr int STREAM_STAGES = 4;
constexpr int STREAM_COLS = 32;

template <typename AT, typename WT, int MR, bool GLU>
constexpr size_t stream_smem() {
  return (size_t)STREAM_STAGES * ((GLU ? 2 : 1) * STREAM_COLS * (STREAM_K * sizeof(WT) + 16) + MR * STREAM_K * sizeof(AT));
}

// The first MR of a block's eight warps multiply, all of them fetch: one or two warps alone spent longer on a stage's 16 to 32
// copies a lane than on its chain (K = 2,048: a row of 2,048 columns 26.6 -> 18.4 us, two 20.5 -> 16.4; two of 32,768 columns,
// bound by memory, 72 -> 70).  Twelve stages instead of four were slower (two rows 20.5 -> 26.6).
constexpr int STREAM_THREADS = 256;

template <typename AT, typename WT, typename OT, int MR, bool GLU>
__global__ void __launch_bounds__(STREAM_THREADS) gemm_stream_kernel(GemmArgs a) {
  constexpr int WARPS = MR < 8 ? MR : 8, R = MR / WARPS, THREADS = STREAM_THREADS;
  constexpr int HALVES = GLU ? 2 : 1, WROWS = HALVES * STREAM_COLS;
  constexpr int WROW = STREAM_K * sizeof(WT) + 16, AROW = STREAM_K * sizeof(AT);
  constexpr int WPIECES = STREAM_K * sizeof(WT) / 16, APIECES = AROW / 16;       // 16-byte pieces of a row
  constexpr int STAGE = WROWS * WROW + MR * AROW;
  extern __shared__ __align__(16) unsigned char stream_sm[];
  __shared__ int tile_info[3];
  if (a.group_offsets || !a.ahead) pdl_wait_only();
  find_tile<MR>(a, tile_info);
  __syncthreads();
  const int group = tile_info[0], row0 = tile_info[1], rows = tile_info[2];
  if (rows <= 0) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n0 = blockIdx.y * STREAM_COLS;
  const AT* A = (const AT*)a.A + (size_t)blockIdx.z * a.a_batch_stride;
  const WT* W = (const WT*)a.W + (size_t)group * a.w_group_stride + (size_t)blockIdx.z * a.w_batch_stride;

  // Rows beyond the last repeat it; columns beyond the last repeat the first ones, spread out (hundreds of blocks that
  // all fetched one row of eight 25 times stood in each other's way: 4,096 rows of 8 columns, K = 512, 34 us); k stops at K.
  const int here = min(a.N - n0, STREAM_COLS), spread = (1 << (31 - __clz(here))) - 1;
  auto fetch_weights = [&](int stage, int k0) {
    unsigned char* to = stream_sm + stage * STAGE;
#pragma unroll
    for (int i = threadIdx.x; i < WROWS * WPIECES; i += THREADS) {
      const int n = i / WPIECES, piece = i % WPIECES, k = k0 + piece * (16 / (int)sizeof(WT)), c = n % STREAM_COLS;
      const int col = n0 + (c < here ? c : c & spread) + (n / STREAM_COLS) * a.N;
      if (k < a.K) cp_async16(to + n * WROW + piece * 16, W + (size_t)col * a.K + k);
    }
  };
  auto fetch_rows = [&](int stage, int k0) {
    unsigned char* to = stream_sm + stage * STAGE + WROWS * WROW;
    for (int i = threadIdx.x; i < MR * APIECES; i += THREADS) {
      const int r = i / APIECES, piece = i % APIECES, k = k0 + piece * (16 / (int)sizeof(AT));
      const int at = row0 + min(r, rows - 1);
      const int src = a.a_rows ? a.a_rows[at] : at;
      if (k < a.K) cp_async16(to + r * AROW + piece * 16, A + (size_t)src * a.lda + k);
    }
  };

  float acc[HALVES][R];
#pragma unroll
  for (int h = 0; h < HALVES; ++h)
#pragma unroll
    for (int r = 0; r < R; ++r) acc[h][r] = 0.f;
  // Nobody writes weights: a dense product's first stages of them are fetched ahead of the wait.
#pragma unroll
  for (int s = 0; s < STREAM_STAGES - 1; ++s)
    if (s * STREAM_K < a.K) fetch_weights(s, s * STREAM_K);
  if (!a.group_offsets) pdl_wait_only();
#pragma unroll
  for (int s = 0; s < STREAM_STAGES - 1; ++s) {
    if (s * STREAM_K < a.K) fetch_rows(s, s * STREAM_K);
    cp_async_commit();
  }
  int stage = 0;
  for (int k0 = 0; k0 < a.K; k0 += STREAM_K) {
    cp_async_wait<STREAM_STAGES - 2>();
    __syncthreads();                           // this stage has landed for all; the one before it is free
    const int ahead = k0 + (STREAM_STAGES - 1) * STREAM_K;
    if (ahead < a.K) {
      fetch_weights((stage + STREAM_STAGES - 1) % STREAM_STAGES, ahead);
      fetch_rows((stage + STREAM_STAGES - 1) % STREAM_STAGES, ahead);
    }
    cp_async_commit();
    const unsigned char* from = stream_sm + stage * STAGE;
    const WT* ws = reinterpret_cast<const WT*>(from + lane * WROW);
    const WT* us = reinterpret_cast<const WT*>(from + (STREAM_COLS + lane) * WROW);
    const AT* as = reinterpret_cast<const AT*>(from + WROWS * WROW) + warp * R * STREAM_K;
    struct Eight { float w[HALVES][8], x[R][8]; };
    auto load = [&](int kk, Eight& e) {
      load8(ws + kk, e.w[0]);
      if constexpr (GLU) load8(us + kk, e.w[HALVES - 1]);
#pragma unroll
      for (int r = 0; r < R; ++r) load8(as + r * STREAM_K + kk, e.x[r]);
    };
    auto add = [&](const Eight& e) {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int h = 0; h < HALVES; ++h) acc[h][r] = fmaf(e.x[r][i], e.w[h][i], acc[h][r]);
    };
    if (warp < WARPS) {
      Eight e[2];
      load(0, e[0]);
      if (k0 + STREAM_K <= a.K) {
#pragma unroll
        for (int kk = 0; kk < STREAM_K; kk += 8) {      // the next eight are read before these are added
          if (kk + 8 < STREAM_K) load(kk + 8, e[(kk / 8 + 1) & 1]);
          add(e[kk / 8 & 1]);
        }
      } else {
        for (int kk = 0; kk < a.K - k0; kk += 8) {
          load(kk, e[0]);
          add(e[0]);
        }
      }
    }
    stage = (stage + 1) % STREAM_STAGES;
  }
  cp_async_wait<0>();
  OT* C = (OT*)a.C + (size_t)blockIdx.z * a.c_batch_stride;
  const int n = n0 + lane;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int at = warp * R + r;
    if (warp < WARPS && at < rows && n < a.N)
      store_out<OT, GLU>(a, C, a.c_rows ? a.c_rows[row0 + at] : row0 + at, n, acc[0][r], acc[HALVES - 1][r]);
  }
}

// Many rows: bound by the multiply-adds (72 TFLOP/s of them on this chip) and by what shared memory returns to
// registers, 128 bytes a cycle whatever is broadcast: 8 x 8 outputs a thread need 16 cycles of it for 16 of
// arithmetic a warp and k, 4 x 8 need 12 for 8.  A block takes 64 rows by 128 weight rows (GLU: 64 gate rows and the
// 64 up rows of the same features), a thread 8 rows by 4 + 4 columns, two multiply-adds an instruction.  A block is
// often alone on its SM with one warp a scheduler (a chain over k can't be split), so nothing hides a latency but
// the thread itself: the next k's operands are read from shared memory before this k's products, the tile after
// next is on its way in registers.  Measured against 4 x 8 outputs with twice the threads: gate_up + GLU of 684 rows
// over 8 experts, 2 x 2688 x 2048, 512 instead of 602 us (the plain kernel: 1,124), 1024 x 4096 x 2048 in 427 instead
// of 454 us (40 TFLOP/s), 342 x 3072 x 2048 level at 124 (161 with the tiles of 64 x 64 before them).  Tried and
// slower: 8 x 8 without the operands read ahead (158 us for the last), 32 rows a block (158), two tiles ahead (175).
template <typename AT, typename WT, typename OT, bool GLU>
__global__ void __launch_bounds__(128) gemm_tile_kernel(GemmArgs a) {
  constexpr int TBM = 64, TBN = 128, TBK = 16, HALF = 64;
  __shared__ __align__(16) float As[2][TBK][TBM];
  __shared__ __align__(16) float Ws[2][TBK][TBN];
  __shared__ int tile_info[3];
  pdl_wait_only();
  find_tile<TBM>(a, tile_info);
  __syncthreads();
  const int group = tile_info[0], row0 = tile_info[1], rows = tile_info[2];
  if (rows <= 0) return;
  const int n0 = blockIdx.y * (GLU ? HALF : TBN);
  const AT* A = (const AT*)a.A + (size_t)blockIdx.z * a.a_batch_stride;
  const WT* W = (const WT*)a.W + (size_t)group * a.w_group_stride + (size_t)blockIdx.z * a.w_batch_stride;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  // this thread loads eight k of row ar and sixteen of weight row threadIdx.x; rows beyond the last repeat it
  const int ar = threadIdx.x & 63, ak = (threadIdx.x >> 6) * 8, wr = threadIdx.x;
  const int at = row0 + min(ar, rows - 1);
  const AT* ap = A + (size_t)(a.a_rows ? a.a_rows[at] : at) * a.lda + ak;
  const int col = GLU ? min(n0 + (wr & (HALF - 1)), a.N - 1) + (wr >= HALF ? a.N : 0) : min(n0 + wr, a.N - 1);
  const WT* wp = W + (size_t)col * a.K;
  unsigned long long acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  __align__(16) AT araw[8];
  __align__(16) WT wraw[16];
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < 8 * (int)sizeof(AT) / 16; ++i)
      reinterpret_cast<uint4*>(araw)[i] = reinterpret_cast<const uint4*>(ap + k0)[i];
#pragma unroll
    for (int i = 0; i < 16 * (int)sizeof(WT) / 16; ++i)
      reinterpret_cast<uint4*>(wraw)[i] = reinterpret_cast<const uint4*>(wp + k0)[i];
  };
  auto put = [&](int b) {
#pragma unroll
    for (int i = 0; i < 8; ++i) As[b][ak + i][ar] = to_float(araw[i]);
#pragma unroll
    for (int i = 0; i < 16; ++i) Ws[b][i][wr] = to_float(wraw[i]);
  };
  struct Frag { float x[8]; ulonglong2 w0, w1; };
  auto frag = [&](int b, int kk, Frag& f) {
    load8(&As[b][kk][ty * 8], f.x);
    f.w0 = *reinterpret_cast<const ulonglong2*>(&Ws[b][kk][tx * 4]);
    f.w1 = *reinterpret_cast<const ulonglong2*>(&Ws[b][kk][HALF + tx * 4]);
  };
  auto mul = [&](const Frag& f) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const unsigned long long x2 = pack2(f.x[i], f.x[i]);
      fma2(acc[i][0], x2, f.w0.x);
      fma2(acc[i][1], x2, f.w0.y);
      fma2(acc[i][2], x2, f.w1.x);
      fma2(acc[i][3], x2, f.w1.y);
    }
  };
  fetch(0);
  put(0);
  if (TBK < a.K) fetch(TBK);
  __syncthreads();
  Frag cur, nxt;
  frag(0, 0, cur);
  int b = 0;
  for (int k0 = 0; k0 < a.K; k0 += TBK, b ^= 1) {
    const bool more = k0 + TBK < a.K;
#pragma unroll
    for (int kk = 0; kk < TBK; ++kk) {
      if (kk + 1 < TBK) frag(b, kk + 1, nxt);
      if (kk == 4 && more) {
        put(b ^ 1);
        if (k0 + 2 * TBK < a.K) fetch(k0 + 2 * TBK);
      }
      if (kk + 1 == TBK) {
        __syncthreads();
        if (more) frag(b ^ 1, 0, nxt);
      }
      mul(cur);
      cur = nxt;
    }
  }
  OT* C = (OT*)a.C + (size_t)blockIdx.z * a.c_batch_stride;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = ty * 8 + i;
    if (r >= rows) continue;
    const int crow = a.c_rows ? a.c_rows[row0 + r] : row0 + r;
    float v[8];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = unpack2(acc[i][j]);
      v[2 * j] = f.x;
      v[2 * j + 1] = f.y;
    }
#pragma unroll
    for (int j = 0; j < (GLU ? 4 : 8); ++j) {
      const int n = n0 + tx * 4 + (j & 3) + (j >= 4 ? HALF : 0);
      if (n < a.N) store_out<OT, GLU>(a, C, crow, n, v[j], v[(j & 3) + 4]);
    }
  }
}

// Dense products whose tiles of 64 x 64 find an SM each: twice as many blocks as above, twice as many threads; 16-byte
// global loads, k-major shared tiles, 128-bit shared loads, the next tile on its way meanwhile.  K % 32 == 0.
template <typename AT, typename WT, typename OT>
__global__ void __launch_bounds__(256) gemm_dense_kernel(GemmArgs a) {
  constexpr int TBM = 64, TBN = 64, TBK = 32;
  __shared__ __align__(16) float As[TBK][TBM + 4];
  __shared__ __align__(16) float Ws[TBK][TBN + 4];
  pdl_wait_only();
  const int row0 = blockIdx.x * TBM, n0 = blockIdx.y * TBN;
  const AT* A = (const AT*)a.A + (size_t)blockIdx.z * a.a_batch_stride;
  const WT* W = (const WT*)a.W + (size_t)blockIdx.z * a.w_batch_stride;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int lr = threadIdx.x >> 2, lk = (threadIdx.x & 3) * 8;      // this thread loads row lr, k lk..lk+7
  const bool a_ok = row0 + lr < a.M, w_ok = n0 + lr < a.N;
  const AT* ap = A + (size_t)(a_ok ? row0 + lr : 0) * a.lda + lk;
  const WT* wp = W + (size_t)(w_ok ? n0 + lr : 0) * a.K + lk;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  float av[8], wv[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) av[i] = wv[i] = 0.f;
  if (a_ok) load8(ap, av);
  if (w_ok) load8(wp, wv);
  for (int k0 = 0; k0 < a.K; k0 += TBK) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      As[lk + i][lr] = av[i];
      Ws[lk + i][lr] = wv[i];
    }
    __syncthreads();
    if (k0 + TBK < a.K) {            // next tile's loads fly while this one is multiplied
      if (a_ok) load8(ap + k0 + TBK, av);
      if (w_ok) load8(wp + k0 + TBK, wv);
    }
#pragma unroll
    for (int kk = 0; kk < TBK; ++kk) {
      const float4 a4 = *reinterpret_cast<const float4*>(&As[kk][ty * 4]);
      const float4 w4 = *reinterpret_cast<const float4*>(&Ws[kk][tx * 4]);
      const float ar[4] = {a4.x, a4.y, a4.z, a4.w}, wr[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(ar[i], wr[j], acc[i][j]);
    }
    __syncthreads();
  }
  OT* C = (OT*)a.C + (size_t)blockIdx.z * a.c_batch_stride;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = row0 + ty * 4 + i;
    if (r >= a.M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < a.N) C[(size_t)r * a.ldc + n] = from_float<OT>(acc[i][j]);
    }
  }
}

template <typename AT, typename WT, typename OT, int MR, bool GLU>
int launch_stream(const GemmArgs& a, cudaStream_t stream) {
  constexpr size_t smem = stream_smem<AT, WT, MR, GLU>();
  const auto kernel = gemm_stream_kernel<AT, WT, OT, MR, GLU>;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  const int tiles = a.group_offsets ? a.M / MR + min(a.G, a.M) : (a.M + MR - 1) / MR;
  const dim3 grid(tiles, (a.N + STREAM_COLS - 1) / STREAM_COLS, a.batch);
  const dim3 block(STREAM_THREADS);
  const cudaError_t e = a.group_offsets ? launch_behind(kernel, grid, block, smem, stream, a)
                                        : launch_pdl(kernel, grid, block, smem, stream, a);
  return e == cudaSuccess ? FT_OK : (int)e;
}

// Which kernel takes a product of M rows (`grouped`: M over G groups), N columns and K, `batch` of them.  Dense ones go
// to the least estimate of time: rounds of blocks on 148 SMs times what a round took per k (0.1 ns; measured over M = 64 ..
// 4,096, N = 8 .. 3,072, K = 64 .. 2,048: the choice is 0.6 % behind the best of the four on average).  gemm_stream_kernel
// reads the weights again for every 16 rows and wins while few blocks share an SM (64 rows, K = N = 2,048: 36 us, tiles of
// 64 x 64 93); gemm_dense_kernel's tiles give twice as many blocks as gemm_tile_kernel's and win where those fit one round
// (2,048 x 256, K = 512: 26 us, 34 and 32), gemm_tile_kernel beyond (1,024 x 4,096, K = 2,048: 427 us); gemm_rows_kernel takes
// many tiles of a K that is no multiple of 16 (2,048 x 4,096, K = 1,000: 694 us, streamed 846).  More columns than a grid's
// second dimension holds blocks of 32 for are not streamed.
enum GemmRoute { GEMM_STREAM, GEMM_TILE, GEMM_DENSE, GEMM_ROWS };
static int gemm_route(int M, int N, int K, int G, int batch, bool grouped, bool glu, bool plain, bool bf16_rows,
                      bool f32_weights) {
  const int half = glu ? 64 : 128;
  const long long wide = (N + half - 1) / half;
  const bool streams = (N + STREAM_COLS - 1) / STREAM_COLS <= 65535;
  if (M / G < 32) return streams ? GEMM_STREAM : GEMM_ROWS;
  // Groups take register tiles from 32 rows each on, where those give half of the SMs a block.
  if (grouped && !(K & 15)) return (M + 63) / 64 * wide >= 64 ? GEMM_TILE : GEMM_STREAM;      // many columns: tiles
  const auto rounds = [](long long blocks) { return (blocks + 147) / 148; };
  const int part = grouped ? G : 0;
  const long long m64 = ((M + 63) / 64 + part) * (long long)batch, narrow = rounds(m64 * ((N + 63) / 64));
  long long best = (f32_weights ? 108 : bf16_rows ? 100 : 85) * (glu ? 2 : 1) *
                   rounds(((M + 15) / 16 + part) * (long long)batch * ((N + STREAM_COLS - 1) / STREAM_COLS)) * (K + 128);
  int route = GEMM_STREAM;
  if (!streams) {
    best = LLONG_MAX;
    route = GEMM_ROWS;
  }
  const auto offer = [&](int r, long long cost) {
    if (cost < best) {
      best = cost;
      route = r;
    }
  };
  if (K & 15) {
    offer(GEMM_ROWS, (780 + 475 * (narrow - 1)) * (glu ? 2 : 1) * (K + 32));
  } else {
    offer(GEMM_TILE, (580 + 500 * (rounds(m64 * wide) - 1)) * (K + 64));
    if (plain && M >= 64 && !(K & 31)) offer(GEMM_DENSE, (453 + 333 * (narrow - 1)) * (K + 56));
  }
  return route;
}

template <typename AT, typename WT, typename OT, bool GLU>
int launch_kind(const GemmArgs& a, cudaStream_t stream) {
  const int per_group = a.group_offsets ? a.M / max(a.G, 1) : a.M;
  const int a_align = sizeof(AT) == 2 ? 7 : 3, w_align = sizeof(WT) == 2 ? 7 : 3;
  const bool pieces = !(a.K & 7) && !(a.lda & a_align) && !(a.a_batch_stride & a_align) &&
                      !(a.w_batch_stride & w_align) && !(a.w_group_stride & w_align) && !((uintptr_t)a.A & 15) &&
                      !((uintptr_t)a.W & 15);
  const bool plain = !GLU && !a.group_offsets && !a.a_rows && !a.c_rows && !a.row_scale;
  const int route = pieces ? gemm_route(a.M, a.N, a.K, a.G, a.batch, a.group_offsets != nullptr, GLU, plain, sizeof(AT) == 2,
                                        sizeof(WT) == 4)
                           : GEMM_ROWS;
  if (route == GEMM_TILE) {
    const int cols = (a.N + (GLU ? 63 : 127)) / (GLU ? 64 : 128);
    const dim3 grid(a.group_offsets ? a.M / 64 + min(a.G, a.M) : (a.M + 63) / 64, cols, a.batch);
    const cudaError_t e = launch_behind(gemm_tile_kernel<AT, WT, OT, GLU>, grid, dim3(128), 0, stream, a);
    return e == cudaSuccess ? FT_OK : (int)e;
  }
  if constexpr (!GLU) {
    if (route == GEMM_DENSE) {
      const cudaError_t e = launch_behind(gemm_dense_kernel<AT, WT, OT>, dim3((a.M + 63) / 64, (a.N + 63) / 64, a.batch), dim3(256),
                                       0, stream, a);
      return e == cudaSuccess ? FT_OK : (int)e;
    }
  }
  if (route == GEMM_STREAM) {
    // rows a block: about twice a group's mean, so that most busy groups are read once
    const int want = a.group_offsets ? 2 * ((a.M + a.G - 1) / a.G) : a.M;
    if (want <= 1) return launch_stream<AT, WT, OT, 1, GLU>(a, stream);
    if (want <= 2) return launch_stream<AT, WT, OT, 2, GLU>(a, stream);
    if (want <= 4) return launch_stream<AT, WT, OT, 4, GLU>(a, stream);
    if (want <= 8) return launch_stream<AT, WT, OT, 8, GLU>(a, stream);
    return launch_stream<AT, WT, OT, 16, GLU>(a, stream);
  }
  const bool big = per_group >= 32;
  const int bm = big ? 64 : 16;
  const int tiles = (a.M + bm - 1) / bm + (a.group_offsets ? a.G : 0);
  const dim3 grid(tiles, (a.N + BN - 1) / BN, a.batch);
  const cudaError_t e = big ? launch_behind(gemm_rows_kernel<AT, WT, OT, 64, GLU>, grid, dim3(256), 0, stream, a)
                            : launch_behind(gemm_rows_kernel<AT, WT, OT, 16, GLU>, grid, dim3(256), 0, stream, a);
  return e == cudaSuccess ? FT_OK : (int)e;
}

template <typename AT, typename WT, typename OT>
int launch(const GemmArgs& a, int glu, cudaStream_t stream) {
  return glu ? launch_kind<AT, WT, OT, true>(a, stream) : launch_kind<AT, WT, OT, false>(a, stream);
}

}  // namespace ft

using namespace ft;

// One dense product per batch entry (a head of a mixer): entry z reads A + z * a_batch_stride
// ([M, K], row stride lda), W + z * w_batch_stride ([N, K]) and writes C + z * c_batch_stride.
extern "C" int ft_gemm_heads(const void* A, int a_dtype, long long lda, long long a_batch_stride, const void* W,
                             int w_dtype, long long w_batch_stride, void* C, int c_dtype, long long ldc,
                             long long c_batch_stride, int M, int N, int K, int batch, cudaStream_t stream);

extern "C" int ft_gemm_route(int M, int N, int K, int G, int batch, int grouped, int glu, int plain, int bf16_rows, int f32_weights) {
  return gemm_route(M, N, K, G, batch, grouped != 0, glu != 0, plain != 0, bf16_rows != 0, f32_weights != 0);
}

// A, W, C element types are given by code; supported triples:
//   (f32,f32,f32) (f32,bf16,f32) (bf16,bf16,bf16) (bf16,bf16,f32) (bf16,f32,f32)
extern "C" int ft_gemm_rows(const void* A, int a_dtype, long long lda, const void* W, int w_dtype,
                            long long w_group_stride, void* C, int c_dtype, long long ldc,
                            const int* group_offsets, const int* a_rows, const int* c_rows,
                            const float* row_scale, int M, int N, int K, int G, int glu, int act,
                            float act_alpha, float act_limit, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return FT_OK;
  if (K <= 0 || G <= 0) return FT_ERR_SHAPE;
  GemmArgs a{A, W, C, group_offsets, a_rows, c_rows, row_scale, lda, ldc, w_group_stride,
             M, N, K, G, act, act_alpha, act_limit};
  a.ahead = promised_ahead;
  const int key = a_dtype * 100 + w_dtype * 10 + c_dtype;
  int rc;
  switch (key) {
    case 0: rc = launch<float, float, float>(a, glu, stream); break;
    case 10: rc = launch<float, __nv_bfloat16, float>(a, glu, stream); break;
    case 111: rc = launch<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(a, glu, stream); break;
    case 110: rc = launch<__nv_bfloat16, __nv_bfloat16, float>(a, glu, stream); break;
    case 100: rc = launch<__nv_bfloat16, float, float>(a, glu, stream); break;
    default: return FT_ERR_DTYPE;
  }
  if (rc != FT_OK) return rc;
  FT_LAUNCH_CHECK();
  return FT_OK;
}

extern "C" int ft_gemm_heads(const void* A, int a_dtype, long long lda, long long a_batch_stride, const void* W,
                             int w_dtype, long long w_batch_stride, void* C, int c_dtype, long long ldc,
                             long long c_batch_stride, int M, int N, int K, int batch, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || batch <= 0) return FT_OK;
  if (K <= 0 || batch > 65535) return FT_ERR_SHAPE;
  GemmArgs a{A, W, C, nullptr, nullptr, nullptr, nullptr, lda, ldc, 0, M, N, K, 1, 0, 0.f, 0.f};
  a.a_batch_stride = a_batch_stride;
  a.w_batch_stride = w_batch_stride;
  a.c_batch_stride = c_batch_stride;
  a.batch = batch;
  a.ahead = promised_ahead;
  const int key = a_dtype * 100 + w_dtype * 10 + c_dtype;
  int rc;
  switch (key) {
    case 0: rc = launch<float, float, float>(a, 0, stream); break;
    case 10: rc = launch<float, __nv_bfloat16, float>(a, 0, stream); break;
    case 111: rc = launch<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(a, 0, stream); break;
    case 110: rc = launch<__nv_bfloat16, __nv_bfloat16, float>(a, 0, stream); break;
    case 100: rc = launch<__nv_bfloat16, float, float>(a, 0, stream); break;
    default: return FT_ERR_DTYPE;
  }
  if (rc != FT_OK) return rc;
  FT_LAUNCH_CHECK();
  return FT_OK;
}

FT_PACKED(ft_gemm_heads)
FT_PACKED(ft_gemm_rows)
