// Shared device helpers for the sm_100a kernels of this package: dtype dispatch, 16-byte vector access, block
// reductions. Launchers are plain `extern "C"` functions taking raw device pointers and a stream, so the library has no
// dependency on torch headers and is loaded from Python with ctypes.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

#include "per_device.h"

#define XL_API extern "C" __attribute__((visibility("default")))

enum XlDtype : int { XL_F32 = 0, XL_F16 = 1, XL_BF16 = 2 };

template <typename T> struct XlVec;  // 16 bytes worth of T
template <> struct XlVec<float> { static constexpr int N = 4; };
template <> struct XlVec<__half> { static constexpr int N = 8; };
template <> struct XlVec<__nv_bfloat16> { static constexpr int N = 8; };

__device__ __forceinline__ float xl_to_float(float v) { return v; }
__device__ __forceinline__ float xl_to_float(__half v) { return __half2float(v); }
__device__ __forceinline__ float xl_to_float(__nv_bfloat16 v) { return __bfloat162float(v); }
template <typename T> __device__ __forceinline__ T xl_from_float(float v);
template <> __device__ __forceinline__ float xl_from_float<float>(float v) { return v; }
template <> __device__ __forceinline__ __half xl_from_float<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 xl_from_float<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}

// Load / store N = 16/sizeof(T) consecutive elements through one 128-bit access. `p` must be 16-byte aligned.
template <typename T> __device__ __forceinline__ void xl_load16(const T* __restrict__ p, float (&out)[XlVec<T>::N]) {
  constexpr int N = XlVec<T>::N;
  uint4 raw = *reinterpret_cast<const uint4*>(p);
  const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int i = 0; i < N; ++i) out[i] = xl_to_float(e[i]);
}
template <typename T> __device__ __forceinline__ void xl_store16(T* __restrict__ p, const float (&in)[XlVec<T>::N]) {
  constexpr int N = XlVec<T>::N;
  uint4 raw;
  T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
  for (int i = 0; i < N; ++i) e[i] = xl_from_float<T>(in[i]);
  *reinterpret_cast<uint4*>(p) = raw;
}

// 16 bytes from an address that is aligned to the element only: the one or two aligned 16-byte blocks that hold them, shifted
// together. Every block read holds at least one of the 16 bytes.
template <typename T> __device__ __forceinline__ uint4 xl_load16_any(const T* __restrict__ p) {
  const uint32_t off = (uint32_t)((uintptr_t)p & 15);
  const uint4* a = reinterpret_cast<const uint4*>((uintptr_t)p - off);
  const uint4 lo = a[0];
  if (off == 0) return lo;
  const uint4 hi = a[1];
  uint4 o;  // words off / 4 .. off / 4 + 4 of the eight; the selections are uniform over a row
  uint32_t w0, w1, w2, w3, w4;
  switch (off >> 2) {
    case 0: w0 = lo.x; w1 = lo.y; w2 = lo.z; w3 = lo.w; w4 = hi.x; break;
    case 1: w0 = lo.y; w1 = lo.z; w2 = lo.w; w3 = hi.x; w4 = hi.y; break;
    case 2: w0 = lo.z; w1 = lo.w; w2 = hi.x; w3 = hi.y; w4 = hi.z; break;
    default: w0 = lo.w; w1 = hi.x; w2 = hi.y; w3 = hi.z; w4 = hi.w; break;
  }
  const uint32_t sh = (off & 3) * 8;
  o.x = __funnelshift_r(w0, w1, sh);
  o.y = __funnelshift_r(w1, w2, sh);
  o.z = __funnelshift_r(w2, w3, sh);
  o.w = __funnelshift_r(w3, w4, sh);
  return o;
}

__device__ __forceinline__ float xl_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float xl_warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
// Block-wide sum; `smem` holds >= 32 floats. All threads get the result.
__device__ __forceinline__ float xl_block_sum(float v, float* smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
  v = xl_warp_sum(v);
  __syncthreads();
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  float r = (lane < nwarps) ? smem[lane] : 0.f;
  return xl_warp_sum(r);
}
__device__ __forceinline__ float xl_block_max(float v, float* smem) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
  v = xl_warp_max(v);
  __syncthreads();
  if (lane == 0) smem[warp] = v;
  __syncthreads();
  float r = (lane < nwarps) ? smem[lane] : -INFINITY;
  return xl_warp_max(r);
}

// Gated unit with clamped inputs: g * sigmoid(slope g) * (u + shift) with g = min(gate, limit), u = clamp(up, -limit, limit).
__device__ __forceinline__ float xl_clamped_glu_value(float gate, float up, float limit, float slope, float shift) {
  const float g = fminf(gate, limit), u = fminf(fmaxf(up, -limit), limit);
  return g / (1.f + expf(-slope * g)) * (u + shift);
}

#define XL_DISPATCH_DTYPE(dtype, T, ...)                                     \
  switch (dtype) {                                                           \
    case XL_F32: { using T = float; __VA_ARGS__; break; }                    \
    case XL_F16: { using T = __half; __VA_ARGS__; break; }                   \
    case XL_BF16: { using T = __nv_bfloat16; __VA_ARGS__; break; }           \
    default: return (int)cudaErrorInvalidValue;                              \
  }

static inline int xl_grid_for(long long n_items, int per_block, int max_blocks = 148 * 16) {
  long long b = (n_items + per_block - 1) / per_block;
  if (b < 1) b = 1;
  if (b > max_blocks) b = max_blocks;
  return (int)b;
}

// Dot product of n values in shared memory (16-byte aligned) with a row in global memory, added in order; rows of whole 16-byte
// pieces are read as such, several ahead.
template <typename T> __device__ __forceinline__ float xl_row_dot(const float* a, const T* row, int n) {
  constexpr int V = 16 / sizeof(T);
  float s = 0.f;
  if (n % V == 0 && (((uintptr_t)row) & 15) == 0) {
#pragma unroll 8
    for (int d = 0; d < n; d += V) {
      const uint4 raw = *reinterpret_cast<const uint4*>(row + d);
      const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
      for (int i = 0; i < V; ++i) s = fmaf(a[d + i], xl_to_float(e[i]), s);
    }
  } else {
    for (int d = 0; d < n; ++d) s = fmaf(a[d], xl_to_float(row[d]), s);
  }
  return s;
}

// Contiguous ranges of items for the CTAs of a grid: the first `rem` CTAs take per + 1 items, the others per.
struct XlRanges {
  int per, rem;
  __device__ __forceinline__ int begin(int cta) const { return cta * per + min(cta, rem); }
  __device__ __forceinline__ int owner(int item) const {
    const int head = rem * (per + 1);
    return item < head ? item / (per + 1) : rem + (item - head) / per;
  }
};

__device__ __forceinline__ void xl_cp_async16(void* smem_dst, const void* src, bool on) {
  const int bytes = on ? 16 : 0;  // 0: the destination is zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem_dst)), "l"(src),
               "r"(bytes)
               : "memory");
}

// two packed 16-bit numbers of type T, low half first
template <typename T> __device__ __forceinline__ float2 xl_pair_to_float2(uint32_t w);
template <> __device__ __forceinline__ float2 xl_pair_to_float2<__half>(uint32_t w) {
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <> __device__ __forceinline__ float2 xl_pair_to_float2<__nv_bfloat16>(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

// Programmatic dependent launch: the kernel may start while its predecessor on the stream drains. It must call
// xl_grid_dependency_wait() before it touches anything the predecessor reads or writes. Operands that were complete before the
// predecessor started (weights, as a rule) may be read ahead of that wait, which hides their latency in the predecessor's tail;
// whether an operand was is the caller's knowledge: such kernels take a `read_ahead` argument, and with 0 they wait first.
// xl_grid_launch_dependents() after that wait lets the successor do the same, so at most two kernels of a chain are in flight. Both are
// no-ops in an ordinary launch, where a kernel may call xl_grid_launch_dependents() at once: it started when all work before it had ended
// (element-wise and attention kernels do, for the products behind them, whose start-up of barriers, TMEM and descriptors takes 2 us
// otherwise). A kernel that allocates TMEM calls it behind the barrier that follows its allocation: a successor allocates before it
// waits, and if its CTA came first on an SM, its columns would wait for this kernel's end and this kernel for its columns.
// No pointer of such a kernel is `__restrict__`: through one, the compiler could move a read of the predecessor's results over the wait.
__device__ __forceinline__ void xl_grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void xl_grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// returns from a launcher whose launch failed
#define XL_TRY(call)                          \
  do {                                        \
    const cudaError_t xl_e = (call);          \
    if (xl_e != cudaSuccess) return (int)xl_e; \
  } while (0)
// Lets launches of `kernel` on the current device take `bytes` of dynamic shared memory. `granted`: what each device allows already.
template <typename K> static inline cudaError_t xl_allow_smem(K kernel, int bytes, XlPerDevice& granted) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess || granted.get(device) >= bytes) return e;
  static std::mutex one_at_a_time;  // the attribute and what is known of it change together
  const std::lock_guard<std::mutex> lock(one_at_a_time);
  if (granted.get(device) >= bytes) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) granted.set(device, bytes);
  return e;
}
template <typename... P, typename... A>
static inline cudaError_t xl_launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
