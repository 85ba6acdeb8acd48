// Causal GQA softmax attention over the paged cache on CUDA cores.
//
// One warp owns one (token, query head).  It walks the keys in chunks of 32
// that are aligned to absolute positions (chunk c = keys 32c..32c+31), keeps a
// running max / sum / accumulator in float32 and visits keys in ascending
// order inside each chunk.  The arithmetic for a (token, head) therefore does
// not depend on whether the token came in a long prompt portion, a two-token
// portion or alone as a decode token, nor on which pages hold the keys.  This
// is the float32 path's attention and the fallback for head sizes the
// tensor-core kernels refuse.
//
// Formula (python/freetoken/kernel/triton/attention.py:74,118-139): scores
// q.k * scale for keys j <= pos (and j > pos - window when a window is set),
// softmax over them, weighted sum of v; query head h reads KV head h / group.
// Options no model of the reference has: a mask in chunks (a query sees the keys
// of its own chunk: floor(j / chunk) == floor(pos / chunk)), scores capped
// as cap * tanh(s / cap), and a sink - a score without key or value that enters
// the softmax's denominator only, fixed (sink_mode 1) or one per query head (2).
//
// Two kernels with the same arithmetic.  attn_shared_kernel brings a chunk's keys and values into shared
// memory once for all the (token, head) rows of a block that read them; attn_paged_kernel reads them from
// global memory row by row (head sizes above 256, rows that are no multiple of 16 bytes).
#include "common.cuh"
#include "mma_utils.cuh"

namespace ft {

struct AttnArgs {
  const void* q;          // [T, nq*d]
  void* out;              // [T, nq*d]
  const void* kv_pages;   // [2, pages, nkv, P, d]
  const int* token_pos;   // [T]
  const int* token_seg;   // [T]
  const int* block_table; // [S, table_width]
  const int* rows;        // token rows to process, or nullptr for 0..T-1
  long long page_stride, kv_stride;
  int nq, nkv, d, P, table_width, window;  // window <= 0: none
  float scale;
  int chunk;              // > 0: keys of the query's own chunk of this many positions only
  float softcap;          // > 0: score <- softcap * tanh(score / softcap)
  int sink_mode;          // 0 none, 1 the score sink_value, 2 sink[h]
  float sink_value;
  const float* sink;      // [nq]
  const int* seg_q_start; // [S + 1] first token of every request, or nullptr
};

// MAXD: output dims per lane (head sizes up to 32 * MAXD)
template <typename AT, bool EXACT, int MAXD>
__global__ void __launch_bounds__(128) attn_paged_kernel(AttnArgs a) {
  extern __shared__ float qs[];  // [4 warps][d]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = a.rows ? a.rows[blockIdx.x] : blockIdx.x;
  const int h = blockIdx.y * 4 + warp;
  if (h >= a.nq) return;
  const int kvh = h / (a.nq / a.nkv);
  const int d = a.d;
  float* qv = qs + warp * d;
  const AT* q = (const AT*)a.q + ((size_t)t * a.nq + h) * d;
  for (int i = lane; i < d; i += 32) qv[i] = to_float(q[i]);
  __syncwarp();

  const int pos = a.token_pos[t];
  const int* table = a.block_table + (size_t)a.token_seg[t] * a.table_width;
  int lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
  if (a.chunk > 0) lo = max(lo, pos - pos % a.chunk);
  const AT* kbase = (const AT*)a.kv_pages + (size_t)kvh * a.P * d;
  const AT* vbase = kbase + a.kv_stride;

  float acc[MAXD];
#pragma unroll
  for (int c = 0; c < MAXD; ++c) acc[c] = 0.f;
  float m = -INFINITY, l = 0.f;

  for (int c0 = (lo / 32) * 32; c0 <= pos; c0 += 32) {
    const int j = c0 + lane;
    const bool valid = j >= lo && j <= pos;
    float s = -INFINITY;
    if (valid) {
      const int page = table[j / a.P];
      const AT* kr = kbase + (size_t)page * a.page_stride + (size_t)(j % a.P) * d;
      float dot = 0.f;
      for (int i = 0; i < d; ++i) dot = fmaf(qv[i], to_float(kr[i]), dot);
      s = dot * a.scale;
      if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
    }
    const float m_new = fmaxf(m, warp_max(s));
    const float p = valid ? (EXACT ? expf(s - m_new) : __expf(s - m_new)) : 0.f;
    const float alpha = (m == -INFINITY) ? 0.f : (EXACT ? expf(m - m_new) : __expf(m - m_new));
    l = l * alpha + warp_sum(p);
    m = m_new;
#pragma unroll
    for (int c = 0; c < MAXD; ++c) acc[c] *= alpha;
    const int jj_lo = max(lo - c0, 0), jj_hi = min(pos - c0, 31);
    for (int jj = jj_lo; jj <= jj_hi; ++jj) {
      const float pj = __shfl_sync(0xffffffffu, p, jj);
      const int jk = c0 + jj;
      const int page = table[jk / a.P];
      const AT* vr = vbase + (size_t)page * a.page_stride + (size_t)(jk % a.P) * d;
#pragma unroll
      for (int c = 0; c < MAXD; ++c) {
        const int i = lane + 32 * c;
        if (i < d) acc[c] = fmaf(pj, to_float(vr[i]), acc[c]);
      }
    }
  }
  if (a.sink_mode) {
    // the sink joins the denominator once, after all keys (so the keys' order of summation
    // does not depend on it)
    const float sk = a.sink_mode == 2 ? a.sink[h] : a.sink_value;
    const float m_new = fmaxf(m, sk);
    const float alpha = EXACT ? expf(m - m_new) : __expf(m - m_new);
    l = l * alpha + (EXACT ? expf(sk - m_new) : __expf(sk - m_new));
#pragma unroll
    for (int c = 0; c < MAXD; ++c) acc[c] *= alpha;
  }
  AT* o = (AT*)a.out + ((size_t)t * a.nq + h) * d;
  const float inv = 1.f / l;
#pragma unroll
  for (int c = 0; c < MAXD; ++c) {
    const int i = lane + 32 * c;
    if (i < d) o[i] = from_float<AT>(acc[c] * inv);
  }
}

// A block's eight warps are (token, query head) rows of one KV head and one request: `tokens` tokens by `heads`
// heads.  They walk the chunks together: every chunk is fetched once by all threads (cp.async, 16-byte
// pieces, the next chunk on its way while this one is used), and a warp leaves out the chunks that its own
// token does not see, so its arithmetic is attn_paged_kernel's, operation by operation.  That kernel is bound
// by latency: a lane reads its key's row from global memory value by value.
// Blocks of several tokens begin every `tokens` tokens (`packs` of them) and end at their request's last token; the
// first tokens of a request that begins inside one have a block of their own (blockIdx.x >= packs).
// Measured (16 heads of 128 on 4 KV heads, float32): two prompts of 214 and 128 tokens in 70 us, a token behind
// each in 25; four launches of the one and sixteen of the other took 4,552 us and take 686.
constexpr int SHARED_WARPS = 8;

__device__ __forceinline__ void piece_of(const float* p, float (&v)[4]) {
  const float4 f = *reinterpret_cast<const float4*>(p);
  v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
}
__device__ __forceinline__ void piece_of(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __bfloat1622float2(h[i]);
    v[2 * i] = f.x;
    v[2 * i + 1] = f.y;
  }
}

template <typename AT, bool EXACT>
__global__ void __launch_bounds__(32 * SHARED_WARPS) attn_shared_kernel(AttnArgs a, int T, int tokens, int heads, int packs) {
  constexpr int MAXD = 8, PIECE = 16 / sizeof(AT), CHUNK = 32;
  extern __shared__ __align__(16) unsigned char sm[];
  __shared__ int row_lo[SHARED_WARPS], row_pos[SHARED_WARPS];
  pdl_wait_only();
  int r_begin = blockIdx.x * tokens, r_end = min(T, r_begin + tokens);
  if ((int)blockIdx.x >= packs) {              // request blockIdx.x - packs + 1, up to where the next pack begins
    const int s = blockIdx.x - packs + 1;
    r_begin = a.seg_q_start[s];
    r_end = min(min((r_begin / tokens + 1) * tokens, a.seg_q_start[s + 1]), T);
    if (r_begin % tokens == 0 || r_end <= r_begin) return;
  } else if (a.seg_q_start) {
    r_end = min(r_end, a.seg_q_start[a.token_seg[r_begin] + 1]);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int d = a.d, group = a.nq / a.nkv, slices = (group + heads - 1) / heads;
  const int krow = d * sizeof(AT) + 16, vrow = d * sizeof(AT);       // padded key rows: no bank conflicts
  const int stage_bytes = CHUNK * (krow + vrow);
  float* qv = reinterpret_cast<float*>(sm + 2 * stage_bytes) + warp * d;
  const int kvh = blockIdx.y / slices, in_group = (blockIdx.y % slices) * heads + warp % heads;
  const int r = r_begin + warp / heads;
  const bool live = r < r_end && in_group < group;
  const int h = kvh * group + in_group;
  int t = 0, pos = -1, lo = 0;
  if (live) {
    t = a.rows ? a.rows[r] : r;
    pos = a.token_pos[t];
    lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    if (a.chunk > 0) lo = max(lo, pos - pos % a.chunk);
    const AT* q = (const AT*)a.q + ((size_t)t * a.nq + h) * d;
    for (int i = lane; i < d; i += 32) qv[i] = to_float(q[i]);
  }
  if (lane == 0) {
    row_lo[warp] = live ? lo : INT_MAX;
    row_pos[warp] = pos;
  }
  __syncthreads();

  float acc[MAXD];
#pragma unroll
  for (int c = 0; c < MAXD; ++c) acc[c] = 0.f;
  float m = -INFINITY, l = 0.f;
  const AT* kbase = (const AT*)a.kv_pages + (size_t)kvh * a.P * d;
  const AT* vbase = kbase + a.kv_stride;

  int first = INT_MAX, last = -1;
  for (int w = 0; w < SHARED_WARPS; ++w) {
    first = min(first, row_lo[w]);
    last = max(last, row_pos[w]);
  }
  if (first <= last) {
    const int* table = a.block_table + (size_t)a.token_seg[a.rows ? a.rows[r_begin] : r_begin] * a.table_width;
    auto fetch = [&](int stage, int c0) {      // keys outside first .. last are never read: those repeat one of them
      unsigned char* ks = sm + stage * stage_bytes;
      unsigned char* vs = ks + CHUNK * krow;
      const int pieces = d / PIECE;
#pragma unroll 4
      for (int i = threadIdx.x; i < CHUNK * pieces; i += 32 * SHARED_WARPS) {
        const int jj = i / pieces, piece = i % pieces;
        const int j = min(max(c0 + jj, first), last);
        const size_t at = (size_t)table[j / a.P] * a.page_stride + (size_t)(j % a.P) * d + piece * PIECE;
        cp_async16(ks + jj * krow + piece * 16, kbase + at);
        cp_async16(vs + jj * vrow + piece * 16, vbase + at);
      }
    };
    const int begin = first / CHUNK * CHUNK;
    fetch(0, begin);
    cp_async_commit();
    int stage = 0;
    for (int c0 = begin; c0 <= last; c0 += CHUNK, stage ^= 1) {
      if (c0 + CHUNK <= last) fetch(stage ^ 1, c0 + CHUNK);
      cp_async_commit();
      cp_async_wait<1>();
      __syncthreads();
      if (c0 <= pos && c0 + CHUNK > lo) {
        const unsigned char* ks = sm + stage * stage_bytes;
        const AT* kr = reinterpret_cast<const AT*>(ks + lane * krow);
        const AT* vs = reinterpret_cast<const AT*>(ks + CHUNK * krow);
        const int j = c0 + lane;
        const bool valid = j >= lo && j <= pos;
        float dot = 0.f;
#pragma unroll 4
        for (int i = 0; i < d; i += PIECE) {
          float kv[PIECE];
          piece_of(kr + i, kv);
#pragma unroll
          for (int e = 0; e < PIECE; ++e) dot = fmaf(qv[i + e], kv[e], dot);
        }
        float s = -INFINITY;
        if (valid) {
          s = dot * a.scale;
          if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float p = valid ? (EXACT ? expf(s - m_new) : __expf(s - m_new)) : 0.f;
        const float alpha = (m == -INFINITY) ? 0.f : (EXACT ? expf(m - m_new) : __expf(m - m_new));
        l = l * alpha + warp_sum(p);
        m = m_new;
#pragma unroll
        for (int c = 0; c < MAXD; ++c) acc[c] *= alpha;
        const int jj_lo = max(lo - c0, 0), jj_hi = min(pos - c0, CHUNK - 1);
#pragma unroll 4
        for (int jj = jj_lo; jj <= jj_hi; ++jj) {
          const float pj = __shfl_sync(0xffffffffu, p, jj);
#pragma unroll
          for (int c = 0; c < MAXD; ++c) {
            const int i = lane + 32 * c;
            if (i < d) acc[c] = fmaf(pj, to_float(vs[jj * d + i]), acc[c]);
          }
        }
      }
      __syncthreads();                         // the stage may be written again
    }
    cp_async_wait<0>();
  }
  if (!live) return;
  if (a.sink_mode) {
    const float sk = a.sink_mode == 2 ? a.sink[h] : a.sink_value;
    const float m_new = fmaxf(m, sk);
    const float alpha = EXACT ? expf(m - m_new) : __expf(m - m_new);
    l = l * alpha + (EXACT ? expf(sk - m_new) : __expf(sk - m_new));
#pragma unroll
    for (int c = 0; c < MAXD; ++c) acc[c] *= alpha;
  }
  AT* o = (AT*)a.out + ((size_t)t * a.nq + h) * d;
  const float inv = 1.f / l;
#pragma unroll
  for (int c = 0; c < MAXD; ++c) {
    const int i = lane + 32 * c;
    if (i < d) o[i] = from_float<AT>(acc[c] * inv);
  }
}

// How many tokens share a block of attn_shared_kernel (at most `fit`); T rows of S requests, `rest` blocks a token.
// One while that leaves SMs without a block, or where every request has one token: rows of different requests share no
// key, and packed into one block they were walked one request after the other (64 requests of 200 keys, 8 heads of 64,
// float32: 147 us, apart 27; row by row from global memory 89).  One as well for rows picked out of several requests:
// where each begins is not known then.  Otherwise neighbours share the chunks: a prompt of 512, 16 heads of 128, 221 us
// (651 with a token a block).
static int attn_tokens_per_block(int T, int S, int rest, int fit, bool starts_known) {
  if ((long long)T * rest <= 2 * 148 || T == S || (S > 1 && !starts_known)) return 1;
  return fit;
}

template <typename AT, bool EXACT>
static int launch_shared(AttnArgs a, int T, int S, cudaStream_t stream) {
  const size_t smem = 2 * (size_t)32 * (2 * a.d * sizeof(AT) + 16) + (size_t)SHARED_WARPS * a.d * sizeof(float);
  const auto kernel = attn_shared_kernel<AT, EXACT>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int group = a.nq / a.nkv, heads = min(group, SHARED_WARPS), slices = (group + heads - 1) / heads;
  const int tokens = attn_tokens_per_block(T, S, a.nkv * slices, SHARED_WARPS / heads, a.seg_q_start != nullptr);
  if (tokens == 1 || S == 1) a.seg_q_start = nullptr;
  const int packs = (T + tokens - 1) / tokens;
  const cudaError_t le = launch_pdl(kernel, dim3(packs + (a.seg_q_start ? S - 1 : 0), a.nkv * slices), dim3(32 * SHARED_WARPS),
                                    smem, stream, a, T, tokens, heads, packs);
  return le == cudaSuccess ? FT_OK : (int)le;
}

}  // namespace ft

using namespace ft;

extern "C" int ft_attn_tokens_per_block(int T, int S, int rest, int fit, int starts_known) {
  return attn_tokens_per_block(T, S, rest, fit, starts_known != 0);
}

// S: rows of the block table, or of seg_q_start where it is given (tokens lie request by request then).
extern "C" int ft_attn_paged_simt(const void* q, void* out, const void* kv_pages,
                                  const int* token_pos, const int* token_seg,
                                  const int* block_table, const int* rows,
                                  long long page_stride, long long kv_stride, int nq, int nkv, int d, int P,
                                  int table_width, int window, float scale, int dtype, int T,
                                  int chunk, float softcap, int sink_mode, float sink_value,
                                  const float* sink, const int* seg_q_start, int S, cudaStream_t stream) {
  if (T <= 0) return FT_OK;
  if (d > 1024 || d <= 0 || nkv <= 0 || nq % nkv) return FT_ERR_SHAPE;
  AttnArgs a{q, out, kv_pages, token_pos, token_seg, block_table, rows, page_stride, kv_stride,
             nq, nkv, d, P, table_width, window, scale, chunk, softcap, sink_mode, sink_value, sink,
             rows ? nullptr : seg_q_start};
  if (sink_mode == 2 && !sink) return FT_ERR_SHAPE;
  dim3 grid(T, (nq + 3) / 4);
  const size_t smem = 4 * (size_t)d * sizeof(float);
  if (dtype != FT_DTYPE_F32 && dtype != FT_DTYPE_BF16) return FT_ERR_DTYPE;
  const int in_piece = dtype == FT_DTYPE_F32 ? 3 : 7;              // 16-byte pieces along a row, from its start
  if (d <= 256 && !(d & in_piece) && !(page_stride & in_piece) && !(kv_stride & in_piece) && !((uintptr_t)kv_pages & 15) &&
      (long long)nkv * nq <= 65535) {
    const int rc = dtype == FT_DTYPE_F32 ? launch_shared<float, true>(a, T, S, stream)
                                         : launch_shared<__nv_bfloat16, false>(a, T, S, stream);
    if (rc != FT_OK) return rc;
  } else if (d <= 256) {
    if (dtype == FT_DTYPE_F32) attn_paged_kernel<float, true, 8><<<grid, 128, smem, stream>>>(a);
    else attn_paged_kernel<__nv_bfloat16, false, 8><<<grid, 128, smem, stream>>>(a);
  } else if (d <= 512) {        // a latent that is wider than any head
    if (dtype == FT_DTYPE_F32) attn_paged_kernel<float, true, 16><<<grid, 128, smem, stream>>>(a);
    else attn_paged_kernel<__nv_bfloat16, false, 16><<<grid, 128, smem, stream>>>(a);
  } else {                      // up to 1024: a latent of 512 values and more with a rotated part behind it
    if (dtype == FT_DTYPE_F32) attn_paged_kernel<float, true, 32><<<grid, 128, smem, stream>>>(a);
    else attn_paged_kernel<__nv_bfloat16, false, 32><<<grid, 128, smem, stream>>>(a);
  }
  FT_LAUNCH_CHECK();
  return FT_OK;
}

FT_PACKED(ft_attn_paged_simt)
