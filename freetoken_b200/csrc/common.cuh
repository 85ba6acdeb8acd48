// Shared device helpers: element types, conversions, deterministic reductions.
//
// Element type codes used by every extern "C" launcher: 0 = float, 1 = bfloat16.
// Reductions have a fixed shape (xor-shuffle tree inside a warp, then a serial
// sum over warps), so a result never depends on how many rows a launch holds.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>
#include <utility>

#define FT_DTYPE_F32 0
#define FT_DTYPE_BF16 1

#define FT_OK 0
#define FT_ERR_DTYPE -101
#define FT_ERR_SHAPE -102

// Run BODY with T bound to the element type named by CODE.
#define FT_DISPATCH(CODE, T, ...)                           \
  switch (CODE) {                                           \
    case FT_DTYPE_F32: { using T = float; __VA_ARGS__; } break;           \
    case FT_DTYPE_BF16: { using T = __nv_bfloat16; __VA_ARGS__; } break;  \
    default: return FT_ERR_DTYPE;                           \
  }

#define FT_LAUNCH_CHECK()                                  \
  do {                                                     \
    cudaError_t e__ = cudaGetLastError();                  \
    if (e__ != cudaSuccess) return (int)e__;               \
  } while (0)

namespace ft {

// Programmatic dependent launch: a kernel launched through launch_pdl() may
// become resident while the kernel before it in the stream is still running;
// pdl_wait() holds it until that kernel has completed and its writes are
// visible, and only then lets the kernel behind it in.  So no more than one
// launch waits beside the one that works, and what a kernel does ahead of its
// wait may read whatever the launch right in front of it does not write:
// weights, tables and the step's metadata where the caller promises it
// (promised_ahead), a request's state where it says so of that.  Everything else is touched behind the wait, and a kernel
// whose blocks all leave must have waited in one of them.  Kernels that fill the
// chip with large blocks (float32 tiles, prompt scans and attention) let the
// next one in only as they leave (pdl_wait_only): resident beside them it works
// in what they leave of an SM's L1 and registers (two ragged float32 prompts
// 7.1 -> 8.6 ms).  (With the second
// half at the top of a kernel, ahead of the wait, a whole chain of launches
// becomes resident at once: 1.55 -> 2.00 ms a step.  The reference wraps the
// same griddepcontrol instructions,
// python/freetoken/kernel/csrc/include/freetoken/utils.cuh:43-57.)
__device__ __forceinline__ void pdl_wait_only() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() {
  pdl_wait_only();
  pdl_release();
}
// Such a kernel reads global memory by plain loads: it is resident all through the launch in front, and a `const __restrict__`
// parameter or __ldg makes a load that is defined only for what nobody writes while the kernel runs, and that the compiler
// may move across the wait.
// Loads for the stretch ahead of the wait: they stay where they are written.
__device__ __forceinline__ float4 ld_ahead4(const float* p) {
  float4 v;
  asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float ld_ahead(const float* p) {
  float v;
  asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}
// The line of `p` is asked into this SM's cache, for constants that a kernel reads where it needs them.
__device__ __forceinline__ void warm(const void* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p) : "memory"); }


// What a softmax attention may do to its scores beyond scale and window (every attention
// kernel takes the same five values): a mask in chunks, a cap, a sink.
struct ScoreOpts {
  int chunk;              // > 0: a query sees the keys of its own chunk of this many positions
  float softcap;          // > 0: score <- softcap * tanh(score / softcap)
  int sink_mode;          // 0 none, 1 the score sink_value, 2 sink[query head]
  float sink_value;
  const float* sink;      // [nq] float32
};
// first key position a query at `pos` sees
__device__ __forceinline__ int first_visible(int pos, int window, int chunk) {
  int lo = window > 0 ? max(0, pos - window + 1) : 0;
  if (chunk > 0) lo = max(lo, pos - pos % chunk);
  return lo;
}
__device__ __forceinline__ float cap_score(float s, float cap) { return cap > 0.f ? cap * tanhf(s / cap) : s; }
// The same for the tensor-core kernels' softmax threads, which are short of issue slots: tanh(x) =
// 1 - 2 / (1 + e^(2x)) from one ex2.approx and one fast division (absolute error of the tanh about
// 1e-6, far below what the bfloat16 operands of a score leave; no NaN at either end: e^(2x) = inf
// gives 1, e^(2x) = 0 gives -1).
__device__ __forceinline__ float cap_score_fast(float s, float cap) {
  float e;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(s * (2.885390081777927f / cap)));
  return cap - __fdividef(2.f * cap, 1.f + e);
}
// The sink joins a running softmax state kept in the log2 domain (max m, sum l): returns the
// factor on the accumulator, updates m and l.  `sink_log2` is the sink's score times log2(e).
__device__ __forceinline__ float join_sink_log2(float& m, float& l, float sink_log2) {
  const float mn = fmaxf(m, sink_log2);
  const float al = (m == -INFINITY) ? 0.f : exp2f(m - mn);
  l = l * al + exp2f(sink_log2 - mn);
  m = mn;
  return al;
}

// A kernel whose blocks are one even round of the chip starts behind the launch in front instead: resident before that has
// left the SMs, they gather on the few that have room (float32 tiles behind a norm of 342 rows: 175 -> 199 us).
template <typename... KArgs, typename... Args>
inline cudaError_t launch_behind(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                 Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                              cudaStream_t stream, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// What a device is asked once and then known for, by its ordinal; 0: not asked yet.  (Several threads may ask at once: they
// get the same answer.)
struct PerDevice {
  static constexpr int MOST = 64;
  std::atomic<int> known[MOST] = {};
  template <typename Ask>
  int get(Ask ask) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
      cudaGetLastError();
      return ask(-1);
    }
    if (dev < 0 || dev >= MOST) return ask(dev);
    int n = known[dev].load(std::memory_order_relaxed);
    if (n == 0) known[dev].store(n = ask(dev), std::memory_order_relaxed);
    return n;
  }
};
// Multiprocessors of the current device (148 where there is none).
inline int device_sms() {
  static PerDevice sms;
  return sms.get([](int dev) {
    int n = 0;
    if (dev >= 0 && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0) return n;
    cudaGetLastError();
    return 148;
  });
}

// Whether the caller of a launcher promises that the launch right in front of it writes nothing of what the kernel reads
// ahead of its wait: weights, tables, the step's metadata.  Without that a kernel waits before it reads anything
// (`if (!ahead) pdl_wait();`, the later wait is then passed at once).  The packed form hands it on for the length of its call;
// who calls a launcher directly promises nothing.
inline thread_local bool promised_ahead = false;

// The packed form of an extern "C" launcher: the arguments in an array of 8-byte words (and behind them the promise),
// taken apart by the types of the launcher's own parameters.  FT_PACKED(name), behind the launcher, defines `name_packed`, which the host side calls.
union PackedArg {
  void* p;
  long long i;
  double f;
};
template <typename T> struct Unpack { static T get(const PackedArg& a) { return (T)a.i; } };
template <typename T> struct Unpack<T*> { static T* get(const PackedArg& a) { return (T*)a.p; } };
template <> struct Unpack<float> { static float get(const PackedArg& a) { return (float)a.f; } };
template <typename... P, size_t... I>
inline int call_packed(int (*f)(P...), const PackedArg* a, std::index_sequence<I...>) {
  return f(Unpack<P>::get(a[I])...);
}
template <typename... P>
inline int call_packed(int (*f)(P...), const PackedArg* a) {
  promised_ahead = a[sizeof...(P)].i != 0;
  const int rc = call_packed(f, a, std::index_sequence_for<P...>());
  promised_ahead = false;
  return rc;
}
#define FT_PACKED(NAME) \
  extern "C" int NAME##_packed(const ft::PackedArg* a) { return ft::call_packed(NAME, a); }

__device__ __forceinline__ float to_float(float v) { return v; }
__device__ __forceinline__ float to_float(__nv_bfloat16 v) { return __bfloat162float(v); }

template <typename T> __device__ __forceinline__ T from_float(float v);
template <> __device__ __forceinline__ float from_float<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum over the block; every thread gets the result.  `scratch` holds 33 floats.
// The order is fixed by blockDim alone.
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();  // scratch may still be read from a previous call
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.f;
    for (int w = 0; w < nwarps; ++w) s += scratch[w];
    scratch[32] = s;
  }
  __syncthreads();
  return scratch[32];
}

}  // namespace ft
