// What the scans of the recurrent mixers share (recurrent.cu: the selective state space; delta_scan.cuh: the delta rule
// and retention): sums over a warp, pieces of a state, rows staged for 16 lanes a column, and the rules that choose
// between kernels of equal results.
//
// Everything that enters a recurrence is float32 whatever the activation type:
// step sizes (softplus), decays (exp), gates (sigmoid), unit norms and the state
// itself.  A request's tokens are taken in order; a segment of a step continues
// from the state its request's slot holds and leaves the state there.  A token's
// result depends on its own request alone: on nothing else in the launch, and on
// how the request was cut into steps only through float32 rounding (it is not:
// every token performs the same operations in the same order whatever the cut).
//
// State layout per head: [N or D][P] float32, P contiguous.  A warp owns WC
// columns of a head's state and its lanes split the rows, so a column's dot
// products are one warp reduction; a block's four warps share the tokens of a
// chunk, which all threads stage into shared memory together.  Which WC a launch
// takes depends on the step's shape, never on a token's place in it, and the
// operations on a column are the same for every WC.  Launches whose segments have several
// tokens may take kernels with 16 lanes a column that perform the same operations (seq_scan
// says which).
#pragma once
#include "common.cuh"

namespace ft {

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

// ------------------------------------------------- segments of several tokens
// A prompt portion's tokens are a chain, and ssd_scan_kernel and delta_scan_kernel spend a microsecond and more on four
// of them: 32 lanes a column, five shuffle stages for the unit vectors, five for the column sums, a broadcast.  In
// ssd_seq_kernel and delta_seq_kernel a column
// belongs to 16 lanes; lane l keeps rows l + 32 e and l + 16 + 32 e of CPL columns, sums them in two chains (what
// lanes l and l + 16 sum there) and adds the two, so that four shuffle stages remain and every sum has the bits of
// the former: which of the two a launch takes does not show in the results.  What does not wait for the
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

// Columns a lane of the kernels for several tokens a segment.  Four need fewer shared loads and less staging a
// column, two leave twice as many blocks.  Time with four over time with two, by the columns of a launch (heads, segments),
// states of 128 x 128, one and four segments of 64 and 512 tokens: delta rule 1.3 .. 1.5 at 2,048, 1.08 .. 1.20 at 4,096,
// 0.90 .. 0.95 at 5,120, 0.80 .. 0.95 from 6,144 to 16,384 (level at 10,240, where two fill a round exactly); a decay
// per channel 1.09 .. 1.16 at 4,096, 0.81 at 5,120; retention and the state space 1.1 .. 1.2 at 2,048, 0.88 .. 0.92 at 4,096.
static int seq_columns(int P, int heads, int S) { return (long long)P * heads * S <= 5000 ? 2 : 4; }

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

}  // namespace ft
