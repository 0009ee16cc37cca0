// Few-rows linear of 32-bit models: y[M, N] = a[M, K] * w[N, K]^T in fp32 FMAs, M <= 16, the weights streamed once.
//
// Bound by reading the weights (at most 16 multiply-adds per weight: 4 rows need a fifth of the FMA rate at full bandwidth). A CTA
// takes R weight rows and its 8 warps split K, so that also 1024 rows give every SM work; lanes read 16-byte pieces of all R
// rows at once, and an activation piece serves R rows. The sums of a thread (R * M of them) are added up over the lanes by halving:
// with every exchange a lane keeps half of the values, 32 values cost 31 exchanges and not 160. Sums are fp32 in a fixed order.
// The first pieces of weights that the predecessor does not write are requested while it drains. 4 rows, matrices of 4 to 46 MB of a 1024-wide model:
// 4.7 to 11 us; the library's kernels took 13 to 14 us and a pass of 2.5 us over their partial sums.
#include "common.cuh"

namespace {

constexpr int LF_WARPS = 8;

// V values summed over the warp: v[0 .. V / 32) of a lane are then the sums of the values that start at the returned index (one value
// for V <= 32, the same one in 32 / V lanes).
template <int V> __device__ __forceinline__ int warp_sum_many(float (&v)[V], int lane) {
  int mine = 0;  // index of v[0] among the V values
#pragma unroll
  for (int off = 16, n = V; off > 0; off >>= 1) {
    if (n > 1) {
      n >>= 1;
      const bool upper = lane & off;
      mine += upper ? n : 0;
#pragma unroll
      for (int i = 0; i < V / 2; ++i) {
        if (i < n) {
          const float send = upper ? v[i] : v[i + n], keep = upper ? v[i + n] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
      }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
    }
  }
  return mine;
}

template <int M, int R>
__global__ void __launch_bounds__(LF_WARPS * 32)
    linear_f32_kernel(const float* a, long long lda, const float* w, float* y, long long ldy, int rows, int N, int K,
                      int read_ahead) {
  constexpr int V = M * R, KEEP = V > 32 ? V / 32 : 1;  // values per lane after the exchange
  __shared__ float red[LF_WARPS][V];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * R;
  const float* wr[R];
#pragma unroll
  for (int r = 0; r < R; ++r) wr[r] = w + (long long)min(n0 + r, N - 1) * K;
  int k = (warp * 32 + lane) * 4;
  float4 wv[R];
  auto load_w = [&](int at) {
#pragma unroll
    for (int r = 0; r < R; ++r) wv[r] = at < K ? __ldcs(reinterpret_cast<const float4*>(wr[r] + at)) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  if (!read_ahead) xl_grid_dependency_wait();
  load_w(k);
  xl_grid_dependency_wait();
  xl_grid_launch_dependents();
  float acc[V];
#pragma unroll
  for (int i = 0; i < V; ++i) acc[i] = 0.f;
  while (k < K) {
    float4 cur[R];
#pragma unroll
    for (int r = 0; r < R; ++r) cur[r] = wv[r];
    const int next = k + LF_WARPS * 128;
    load_w(next);
#pragma unroll
    for (int m = 0; m < M; ++m) {
      if (m < rows) {
        const float4 x = *reinterpret_cast<const float4*>(a + m * lda + k);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          float& s = acc[m * R + r];
          s = fmaf(cur[r].x, x.x, s);
          s = fmaf(cur[r].y, x.y, s);
          s = fmaf(cur[r].z, x.z, s);
          s = fmaf(cur[r].w, x.w, s);
        }
      }
    }
    k = next;
  }
  const int mine = warp_sum_many<V>(acc, lane);
#pragma unroll
  for (int i = 0; i < KEEP; ++i) red[warp][mine + i] = acc[i];  // with V < 32 several lanes write the same sum
  __syncthreads();
  for (int i = threadIdx.x; i < V; i += LF_WARPS * 32) {
    float s = 0.f;
#pragma unroll
    for (int v = 0; v < LF_WARPS; ++v) s += red[v][i];
    const int m = i / R, n = n0 + i % R;
    if (m < rows && n < N) y[m * ldy + n] = s;
  }
}

template <int M, int R> int lf_launch(const float* a, long long lda, const float* w, float* y, long long ldy, int rows, int N, int K,
                                     int read_ahead, cudaStream_t s) {
  const cudaError_t e = xl_launch_overlapped(linear_f32_kernel<M, R>, dim3((N + R - 1) / R), dim3(LF_WARPS * 32), (size_t)0, s, a, lda, w, y,
                                             ldy, rows, N, K, read_ahead);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

}  // namespace

// a (M, K) with row stride lda, w (N, K) contiguous, y (M, N) with row stride ldy, all fp32; M <= 16, K and lda multiples of 4, a and w
// 16-byte aligned. read_ahead: w was complete before the previous launch on the stream. Returns -1 for arguments the kernel does not take.
XL_API int xl_linear_f32(const float* a, long long lda, const float* w, float* y, long long ldy, int M, int N, int K, int read_ahead,
                         cudaStream_t s) {
  if (M < 1 || M > 16 || N < 1 || K < 4 || (K % 4) || (lda % 4) || lda < K || (((uintptr_t)a | (uintptr_t)w) & 15) || !y) return -1;
  // eight rows per CTA where that still gives every SM two CTAs: half as many reads of the activations
  const bool wide = N >= 8 * 2 * 148;
  if (M == 1) return wide ? lf_launch<1, 8>(a, lda, w, y, ldy, M, N, K, read_ahead, s) : lf_launch<1, 4>(a, lda, w, y, ldy, M, N, K, read_ahead, s);
  if (M == 2) return wide ? lf_launch<2, 8>(a, lda, w, y, ldy, M, N, K, read_ahead, s) : lf_launch<2, 4>(a, lda, w, y, ldy, M, N, K, read_ahead, s);
  if (M <= 4) return wide ? lf_launch<4, 8>(a, lda, w, y, ldy, M, N, K, read_ahead, s) : lf_launch<4, 4>(a, lda, w, y, ldy, M, N, K, read_ahead, s);
  if (M <= 8) return wide ? lf_launch<8, 8>(a, lda, w, y, ldy, M, N, K, read_ahead, s) : lf_launch<8, 4>(a, lda, w, y, ldy, M, N, K, read_ahead, s);
  return lf_launch<16, 4>(a, lda, w, y, ldy, M, N, K, read_ahead, s);
}
