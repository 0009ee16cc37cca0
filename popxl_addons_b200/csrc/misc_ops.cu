// Smaller device ops of the add-on layer:
//   xl_pow2_cast_to_fp8 / xl_pow2_cast_from_fp8   power-of-two scaled casts between 16/32-bit floats and e4m3 / e5m2
//   xl_fp8_mse_scale                              power-of-two scale that minimises the squared quantisation error
//   xl_dense_csr_matmul                           dense x constant CSR matrix
//   xl_gather_rows / xl_scatter_add_rows          embedding lookup (rows out of range give zeros) and its gradient
//   xl_row_stats / xl_ce_shard_*                  row statistics of hidden-sharded LayerNorm and vocabulary-sharded
//                                                 cross-entropy (the pieces between the small all-reduces)
#include "common.cuh"

#include <cuda_fp8.h>
#include <math.h>

// ------------------------------------------------------------------------------------------------------------------
// FP8 casts. log2_scale is a device scalar (int32 or fp32); y = saturate(x * 2^s) in the 8-bit format, and back.
// ------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float load_log2(const void* p, int is_int) {
  return is_int ? (float)(*(const int*)p) : *(const float*)p;
}

template <typename T>
__global__ void __launch_bounds__(256)
    pow2_cast_to_fp8_kernel(const T* __restrict__ x, const void* __restrict__ log2_scale, int log2_is_int,
                            uint8_t* __restrict__ y, long long n, int e5m2) {
  const float s = exp2f(load_log2(log2_scale, log2_is_int));
  const __nv_fp8_interpretation_t fmt = e5m2 ? __NV_E5M2 : __NV_E4M3;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    y[i] = (uint8_t)__nv_cvt_float_to_fp8(xl_to_float(x[i]) * s, __NV_SATFINITE, fmt);
}

template <typename T>
__global__ void __launch_bounds__(256)
    pow2_cast_from_fp8_kernel(const uint8_t* __restrict__ x, const void* __restrict__ log2_scale, int log2_is_int,
                              T* __restrict__ y, long long n, int e5m2) {
  const float s = exp2f(load_log2(log2_scale, log2_is_int));
  const __nv_fp8_interpretation_t fmt = e5m2 ? __NV_E5M2 : __NV_E4M3;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const __half_raw h = __nv_cvt_fp8_to_halfraw((__nv_fp8_storage_t)x[i], fmt);
    y[i] = xl_from_float<T>(__half2float(__half(h)) * s);
  }
}

XL_API int xl_pow2_cast_to_fp8(const void* x, int dtype, const void* log2_scale, int log2_is_int, void* y, long long n,
                               int e5m2, cudaStream_t s) {
  const int grid = xl_grid_for(n, 256 * 4);
  XL_DISPATCH_DTYPE(dtype, T, {
    pow2_cast_to_fp8_kernel<T><<<grid, 256, 0, s>>>((const T*)x, log2_scale, log2_is_int, (uint8_t*)y, n, e5m2);
  });
  return (int)cudaGetLastError();
}

XL_API int xl_pow2_cast_from_fp8(const void* x, const void* log2_scale, int log2_is_int, void* y, int dtype, long long n,
                                 int e5m2, cudaStream_t s) {
  const int grid = xl_grid_for(n, 256 * 4);
  XL_DISPATCH_DTYPE(dtype, T, {
    pow2_cast_from_fp8_kernel<T><<<grid, 256, 0, s>>>((const uint8_t*)x, log2_scale, log2_is_int, (T*)y, n, e5m2);
  });
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------------------------
// Best power-of-two scale for an 8-bit format by squared error (the algorithm of ops/fp8_mse_scale.py):
// histogram of |x| over the 254 octaves of normal fp32 numbers (shared-memory atomics, then global atomics); the last
// block to finish evaluates the 62 candidate shifts in double precision, writes the result and leaves the scratch
// (254 counters + ticket) zeroed.
// ------------------------------------------------------------------------------------------------------------------
constexpr int MSE_BINS = 254;
constexpr int MSE_CANDIDATES = 62;

template <typename T>
__global__ void __launch_bounds__(256)
    fp8_mse_scale_kernel(const T* __restrict__ x, long long n, unsigned int* __restrict__ scratch, int lo, int span,
                         double qerr, int* __restrict__ out) {
  __shared__ unsigned int hist[MSE_BINS];
  __shared__ double cost[MSE_CANDIDATES];
  __shared__ unsigned int last;
  for (int i = threadIdx.x; i < MSE_BINS; i += blockDim.x) hist[i] = 0;
  __syncthreads();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const unsigned int e = (__float_as_uint(fabsf(xl_to_float(x[i]))) >> 23) & 0xFFu;  // biased exponent
    if (e >= 1 && e <= 254) atomicAdd(&hist[e - 1], 1u);  // zeros and subnormals are not counted; inf / nan ignored
  }
  __syncthreads();
  for (int i = threadIdx.x; i < MSE_BINS; i += blockDim.x)
    if (hist[i]) atomicAdd(&scratch[i], hist[i]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&scratch[MSE_BINS], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (threadIdx.x < MSE_CANDIDATES) {
    const int c = threadIdx.x;
    const int first = lo - 31 + 126;  // bin of the lowest covered octave for the first candidate shift (-31)
    const int start = first + c, stop = first + c + span;
    const int top_bin = min(max(stop - 1, 0), MSE_BINS - 1);
    const double top = exp2((double)(top_bin - 126));
    const double inv_n = 1.0 / (double)(n > 0 ? n : 1);
    double acc_under = 0.0, acc_in = 0.0, acc_over = 0.0;
    for (int b = 0; b < MSE_BINS; ++b) {
      const double h = (double)__ldcg(&scratch[b]) * inv_n;
      const double v = exp2((double)(b - 126));
      if (b < start) { if (b >= 1) acc_under += h * v * v; }
      else if (b < stop) acc_in += h * v * v * qerr;
      else acc_over += h * (v - top) * (v - top);
    }
    cost[c] = acc_under + acc_in + acc_over;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double best = cost[0];
    int arg = 0;
    for (int c = 1; c < MSE_CANDIDATES; ++c)
      if (cost[c] < best) { best = cost[c]; arg = c; }
    int ties = 0;
    for (int c = 0; c < MSE_CANDIDATES; ++c) ties += cost[c] == best;
    *out = -(arg + ties / 2 - 31);
  }
  __syncthreads();
  for (int i = threadIdx.x; i <= MSE_BINS; i += blockDim.x) scratch[i] = 0;
}

// scratch: 255 zero-initialised words (left zeroed). lo / span: lowest octave covered by the format and the number of
// octaves it covers; qerr = 2^(-2 * (source mantissa bits - format mantissa bits)).
XL_API int xl_fp8_mse_scale(const void* x, int dtype, long long n, unsigned int* scratch, int lo, int span, double qerr,
                            int* out, cudaStream_t s) {
  const int grid = xl_grid_for(n, 256 * 8, 148 * 4);
  XL_DISPATCH_DTYPE(dtype, T, {
    fp8_mse_scale_kernel<T><<<grid, 256, 0, s>>>((const T*)x, n, scratch, lo, span, qerr, out);
  });
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------------------------
// y (M, N) = x (M, K) @ S, S a constant K x N matrix in CSR form (indptr K+1, indices, values). One CTA per output row:
// the row is accumulated in shared memory (fp32); threads walk the non-zeros, the CSR row of a non-zero is found by
// bisection of indptr. N * 4 bytes must fit in 48 KB of shared memory.
// ------------------------------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
    dense_csr_matmul_kernel(const T* __restrict__ x, const int* __restrict__ indptr, const int* __restrict__ indices,
                            const float* __restrict__ values, T* __restrict__ y, int K, int N, int nnz) {
  extern __shared__ float acc[];
  const int m = blockIdx.x;
  for (int i = threadIdx.x; i < N; i += blockDim.x) acc[i] = 0.f;
  __syncthreads();
  const T* xr = x + (long long)m * K;
  for (int idx = threadIdx.x; idx < nnz; idx += blockDim.x) {
    int lo = 0, hi = K;  // largest k with indptr[k] <= idx
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (indptr[mid] <= idx) lo = mid;
      else hi = mid;
    }
    atomicAdd(&acc[indices[idx]], xl_to_float(xr[lo]) * values[idx]);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < N; i += blockDim.x) y[(long long)m * N + i] = xl_from_float<T>(acc[i]);
}

XL_API int xl_dense_csr_matmul(const void* x, int dtype, const int* indptr, const int* indices, const float* values, void* y,
                               int M, int K, int N, int nnz, cudaStream_t s) {
  if (M < 1 || N < 1 || (long long)N * 4 > 48 * 1024) return -1;
  XL_DISPATCH_DTYPE(dtype, T, {
    dense_csr_matmul_kernel<T><<<M, 256, N * 4, s>>>((const T*)x, indptr, indices, values, (T*)y, K, N, nnz);
  });
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------------------------
// Embedding lookup on a vocabulary shard: out[i, :] = table[idx[i], :] if 0 <= idx[i] < rows else 0 (zero_oor), and the
// gradient scatter-add into an fp32 or 16-bit table gradient. cols % 8 == 0 for the vector path of 16-bit tables.
// ------------------------------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
    gather_rows_kernel(const T* table, const int* idx, T* out, long long n_idx, int rows, int cols) {
  xl_grid_dependency_wait();
  xl_grid_launch_dependents();
  const long long i = blockIdx.x;
  if (i >= n_idx) return;
  const int r = idx[i];
  const bool ok = r >= 0 && r < rows;
  const T* src = table + (long long)(ok ? r : 0) * cols;
  T* dst = out + i * cols;
  constexpr int V = 16 / sizeof(T);
  if (cols % V == 0 && ((((uintptr_t)table) | ((uintptr_t)out)) & 15) == 0) {
    for (int c = threadIdx.x * V; c < cols; c += blockDim.x * V)
      *reinterpret_cast<uint4*>(dst + c) = ok ? *reinterpret_cast<const uint4*>(src + c) : make_uint4(0, 0, 0, 0);
  } else {
    for (int c = threadIdx.x; c < cols; c += blockDim.x) dst[c] = ok ? src[c] : xl_from_float<T>(0.f);
  }
}

template <typename T, typename G>
__global__ void __launch_bounds__(256)
    scatter_add_rows_kernel(const G* __restrict__ grad_out, const int* __restrict__ idx, T* __restrict__ grad_table,
                            long long n_idx, int rows, int cols) {
  const long long i = blockIdx.x;
  if (i >= n_idx) return;
  const int r = idx[i];
  if (r < 0 || r >= rows) return;
  const G* src = grad_out + i * cols;
  T* dst = grad_table + (long long)r * cols;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) atomicAdd(dst + c, (T)xl_to_float(src[c]));
}

XL_API int xl_gather_rows(const void* table, int dtype, const int* idx, void* out, long long n_idx, int rows, int cols,
                          cudaStream_t s) {
  if (n_idx < 1) return 0;
  XL_DISPATCH_DTYPE(dtype, T, {
    const cudaError_t e = xl_launch_overlapped(gather_rows_kernel<T>, dim3((unsigned)n_idx), dim3(256), (size_t)0, s, (const T*)table, idx,
                                               (T*)out, n_idx, rows, cols);
    if (e != cudaSuccess) return (int)e;
  });
  return (int)cudaGetLastError();
}

// grad_table: fp32 (rows, cols), accumulated into (not zeroed here); grad_out: (n_idx, cols) of dtype.
XL_API int xl_scatter_add_rows(const void* grad_out, int dtype, const int* idx, float* grad_table, long long n_idx, int rows,
                               int cols, cudaStream_t s) {
  if (n_idx < 1) return 0;
  XL_DISPATCH_DTYPE(dtype, G, {
    scatter_add_rows_kernel<float, G><<<(unsigned)n_idx, 256, 0, s>>>((const G*)grad_out, idx, grad_table, n_idx, rows,
                                                                      cols);
  });
  return (int)cudaGetLastError();
}

// V consecutive values of any type as fp32: single ones, or four with one access
template <typename G, int V> __device__ __forceinline__ void xl_load_group(const G* p, float (&out)[V]) {
  if constexpr (V == 1) {
    out[0] = xl_to_float(*p);
  } else if constexpr (sizeof(G) == 4) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
  } else {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    const G* e = reinterpret_cast<const G*>(&v);
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = xl_to_float(e[i]);
  }
}

// Running mean of an embedding table's gradient, without the dense gradient: acc = acc * t/(t+1), then the rows that the tokens
// picked += (sum of their grad_out) / (t+1), t = *step. Bound by the first part, one read and write of the table. The second adds a
// row's tokens up in an order that depends on the indices alone, so that the same inputs give the same bits (atomic additions did not:
// a training step differed from itself by 1e-7). For that the first launch also sorts the tokens by row, in CTAs of its own beside the
// pass over the table: a token's place is the number of tokens with a smaller row, and of earlier ones with the same.
// 50400 x 4096, 2048 tokens: zero fill, scatter, cast and dense running mean took 783 us, a pass and atomic additions 270, this 298;
// 50257 x 768, 4096 tokens 158, 51, 57; 1024 x 256, 256 tokens 7.2, 4.0, 5.2. 8192 tokens of a text (a frequent word has hundreds): 387.
constexpr int EMB_TOKENS = 32768;           // tokens per pair of launches
constexpr int EMB_SORTED = 64;              // tokens a CTA finds the places of, four threads each
constexpr int EMB_NONE = 0x7fffffff;        // the row of a token outside the table: sorted behind all others
__global__ void __launch_bounds__(256)
    mean_decay_and_sort_kernel(float* __restrict__ acc, const float* __restrict__ step, long long n, const int* __restrict__ idx, int n_idx,
                               int rows, int sort_ctas, int* __restrict__ order) {  // order: n_idx sorted rows, n_idx tokens
  xl_grid_launch_dependents();
  if ((int)blockIdx.x < sort_ctas) {
    __shared__ __align__(16) int keys[1024];
    const int first = blockIdx.x * EMB_SORTED, i = first + (threadIdx.x >> 2), q = threadIdx.x & 3;
    auto key = [&](int j) {
      const int r = j < n_idx ? idx[j] : -1;
      return r >= 0 && r < rows ? r : EMB_NONE;
    };
    const int mine = key(i);
    int place = 0;
    for (int base = 0; base < n_idx; base += 1024) {
      __syncthreads();
#pragma unroll
      for (int e = 0; e < 1024; e += 256) keys[e + threadIdx.x] = key(base + e + threadIdx.x);
      __syncthreads();
      // in fours: earlier tokens than the CTA's, the CTA's, later ones
      const int4* k4 = reinterpret_cast<const int4*>(keys);
      const int end = min(256, (n_idx - base + 3) / 4);
      const int own = min(max(first - base, 0) / 4, end), later = min(max(first + EMB_SORTED - base, 0) / 4, end);
#pragma unroll 8
      for (int j = q; j < own; j += 4) {
        const int4 k = k4[j];
        place += (k.x <= mine) + (k.y <= mine) + (k.z <= mine) + (k.w <= mine);
      }
      for (int j = own + q; j < later; j += 4) {
        const int4 k = k4[j];
        const int at = base + 4 * j;
        place += (k.x < mine || (k.x == mine && at < i)) + (k.y < mine || (k.y == mine && at + 1 < i)) +
                 (k.z < mine || (k.z == mine && at + 2 < i)) + (k.w < mine || (k.w == mine && at + 3 < i));
      }
#pragma unroll 8
      for (int j = later + q; j < end; j += 4) {
        const int4 k = k4[j];
        place += (k.x < mine) + (k.y < mine) + (k.z < mine) + (k.w < mine);
      }
    }
    place += __shfl_xor_sync(0xffffffffu, place, 1);
    place += __shfl_xor_sync(0xffffffffu, place, 2);
    if (q == 0 && i < n_idx) {
      order[place] = mine;
      order[n_idx + place] = i;
    }
    return;
  }
  const float t = *step;
  const float a = t / (t + 1.f);
  const long long groups = n / 4;
  float4* acc4 = reinterpret_cast<float4*>(acc);
  const long long cta = blockIdx.x - sort_ctas, stride = (long long)(gridDim.x - sort_ctas) * 256, first = cta * 256 + threadIdx.x;
  for (long long i = first; i < groups; i += 2 * stride) {
    const bool two = i + stride < groups;
    float4 p = __ldcs(acc4 + i), q = two ? __ldcs(acc4 + i + stride) : make_float4(0.f, 0.f, 0.f, 0.f);
    p.x *= a; p.y *= a; p.z *= a; p.w *= a;
    q.x *= a; q.y *= a; q.z *= a; q.w *= a;
    __stcs(acc4 + i, p);
    if (two) __stcs(acc4 + i + stride, q);
  }
  if (first < n - groups * 4) acc[groups * 4 + first] *= a;
}

// A warp takes the tokens of one row (from the place in the sorted list where they begin) and NB times 32 V columns. Rows with 32
// tokens and more (padding, frequent words) are shared by the eight warps of the CTA, an eighth of the tokens each.
template <typename G, int V, int NB>
__global__ void __launch_bounds__(256)
    add_sorted_rows_kernel(const G* __restrict__ grad_out, const int* __restrict__ order, float* __restrict__ acc,
                           const float* __restrict__ step, int n_idx, int cols) {
  xl_grid_launch_dependents();
  constexpr int WIDTH = 32 * V * NB, AHEAD = 8 / NB;
  __shared__ float part[8][WIDTH];
  __shared__ int shared_row[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int place = blockIdx.x * 8 + warp, c = blockIdx.y * WIDTH + lane * V;  // and every 32 V columns on
  const int *order_row = order, *order_token = order + n_idx;
  float sum[NB][V], old[NB][V];
  auto add_tokens = [&](int from, int to, int token) {  // token: of place from + lane
#pragma unroll
    for (int q = 0; q < NB; ++q)
#pragma unroll
      for (int e = 0; e < V; ++e) sum[q][e] = 0.f;
    for (int k0 = from; k0 < to; k0 += 32) {
      const int n = min(32, to - k0);
      if (k0 > from) token = lane < n ? order_token[k0 + lane] : 0;
      for (int k1 = 0; k1 < n; k1 += AHEAD) {
        float g[AHEAD][NB][V];
#pragma unroll
        for (int k = 0; k < AHEAD; ++k) {
          const int tk = __shfl_sync(0xffffffffu, token, (k1 + k) & 31);
#pragma unroll
          for (int q = 0; q < NB; ++q)
            if (k1 + k < n && c + q * 32 * V < cols) xl_load_group<G, V>(grad_out + (long long)tk * cols + c + q * 32 * V, g[k][q]);
        }
#pragma unroll
        for (int k = 0; k < AHEAD; ++k)
          if (k1 + k < n)
#pragma unroll
            for (int q = 0; q < NB; ++q)
#pragma unroll
              for (int e = 0; e < V; ++e) sum[q][e] += g[k][q][e];
      }
    }
  };
  auto load_old = [&](int row) {
#pragma unroll
    for (int q = 0; q < NB; ++q)
      if (c + q * 32 * V < cols) xl_load_group<float, V>(acc + (long long)row * cols + c + q * 32 * V, old[q]);
  };
  const float b = 1.f / (*step + 1.f);
  auto store = [&](int row) {
#pragma unroll
    for (int q = 0; q < NB; ++q) {
      if (c + q * 32 * V >= cols) continue;
      float* dst = acc + (long long)row * cols + c + q * 32 * V;
#pragma unroll
      for (int e = 0; e < V; ++e) old[q][e] += sum[q][e] * b;
      if constexpr (V == 4) *reinterpret_cast<float4*>(dst) = make_float4(old[q][0], old[q][1], old[q][2], old[q][3]);
      else dst[0] = old[q][0];
    }
  };
  // the list around this warp's place, in one go: the row before it, its row and the 31 after, their tokens
  const int at = place + lane;
  const int row_at = at < n_idx ? order_row[at] : EMB_NONE, token = at < n_idx ? order_token[at] : 0;
  const int before = place > 0 && place < n_idx ? order_row[place - 1] : EMB_NONE;
  const int row = __shfl_sync(0xffffffffu, row_at, 0);
  const bool begins = row != EMB_NONE && before != row;
  const unsigned same = __ballot_sync(0xffffffffu, begins && row_at == row);
  const bool shared = same == 0xffffffffu;
  if (begins && !shared) {
    load_old(row);
    add_tokens(place, place + __popc(same), token);
    store(row);
  }
  if (lane == 0) shared_row[warp] = shared ? row : EMB_NONE;
  if (!__syncthreads_or(shared)) return;
  for (int w = 0; w < 8; ++w) {
    const int r = shared_row[w];
    if (r == EMB_NONE) continue;
    const int from = blockIdx.x * 8 + w;
    int last = from + 31, end = n_idx;  // the row's tokens reach up to `last` at least and to before `end`
    while (end - last > 1) {
      const int gap = (end - last + 31) / 32, probe = last + (lane + 1) * gap;
      const unsigned m = __ballot_sync(0xffffffffu, probe < end && order_row[min(probe, n_idx - 1)] == r);
      last += __popc(m) * gap;
      end = min(end, last + gap);
    }
    const int n = last + 1 - from, begin = from + (int)((long long)n * warp / 8), stop = from + (int)((long long)n * (warp + 1) / 8);
    if (warp == 0) load_old(r);
    add_tokens(begin, stop, begin + lane < stop ? order_token[begin + lane] : 0);
#pragma unroll
    for (int q = 0; q < NB; ++q)
#pragma unroll
      for (int e = 0; e < V; ++e) part[warp][(q * 32 + lane) * V + e] = sum[q][e];
    __syncthreads();
    if (warp == 0) {
#pragma unroll
      for (int q = 0; q < NB; ++q)
#pragma unroll
        for (int e = 0; e < V; ++e) {
          sum[q][e] = 0.f;
          for (int v = 0; v < 8; ++v) sum[q][e] += part[v][(q * 32 + lane) * V + e];
        }
      store(r);
    }
    __syncthreads();
  }
}
// Integers of scratch for n_idx tokens.
XL_API long long xl_scatter_mean_scratch(long long n_idx) { return 2 * (n_idx < EMB_TOKENS ? n_idx : EMB_TOKENS); }
// acc: fp32 (rows, cols), contiguous and 16-byte aligned; grad_out: (n_idx, cols) of dtype, aligned likewise. Indices outside the table
// are skipped.
XL_API int xl_scatter_mean_rows(const void* grad_out, int dtype, const int* idx, float* acc, const float* step, long long n_idx,
                                int rows, int cols, int* order, cudaStream_t s) {
  const long long n = (long long)rows * cols;
  if (n < 1) return 0;
  if ((((uintptr_t)acc) | ((uintptr_t)grad_out)) & 15 || (n_idx > 0 && !order)) return -1;
  const int width = cols % 4 ? 32 : cols > 128 ? 256 : 128;  // columns per warp
  if ((cols + width - 1) / width > 65535) return -1;
  for (long long i0 = 0; i0 == 0 || i0 < n_idx; i0 += EMB_TOKENS) {
    const int m = (int)(n_idx - i0 < EMB_TOKENS ? n_idx - i0 : EMB_TOKENS), sort_ctas = (m + EMB_SORTED - 1) / EMB_SORTED;
    const int decay_ctas = i0 == 0 ? xl_grid_for(n, 256 * 8) : 0;  // the mean's old part once
    mean_decay_and_sort_kernel<<<sort_ctas + decay_ctas, 256, 0, s>>>(acc, step, n, idx + i0, m, rows, sort_ctas, order);
    if (m == 0) break;
    const dim3 grid((m + 7) / 8, (cols + width - 1) / width);
    XL_DISPATCH_DTYPE(dtype, G, {
      const G* g = (const G*)grad_out + i0 * cols;
      if (width == 256) add_sorted_rows_kernel<G, 4, 2><<<grid, 256, 0, s>>>(g, order, acc, step, m, cols);
      else if (width == 128) add_sorted_rows_kernel<G, 4, 1><<<grid, 256, 0, s>>>(g, order, acc, step, m, cols);
      else add_sorted_rows_kernel<G, 1, 1><<<grid, 256, 0, s>>>(g, order, acc, step, m, cols);
    });
  }
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------------------------
// Row statistics for ops whose rows are sharded over ranks: per row (sum, sum of squares) for the hidden-sharded
// LayerNorm's forward pass (its backward pass and the vocabulary-sharded cross-entropy are in sharded_ops.cu). The tiny
// per-row results are all-reduced by the caller between the kernels. One CTA per row.
// ------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float block_sum_256(float v, float* red) {
  v = xl_warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.f;
  for (int i = 0; i < 8; ++i) t += red[i];
  return t;
}
__device__ __forceinline__ float block_max_256(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = -INFINITY;
  for (int i = 0; i < 8; ++i) t = fmaxf(t, red[i]);
  return t;
}

// stats: (2, rows) fp32 = [sum | sum of squares]
template <typename T>
__global__ void __launch_bounds__(256) row_sum_sumsq_kernel(const T* __restrict__ x, float* __restrict__ stats, int rows, int cols) {
  __shared__ float red[8];
  const int r = blockIdx.x;
  float s = 0.f, q = 0.f;
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    const float v = xl_to_float(x[(long long)r * cols + c]);
    s += v;
    q += v * v;
  }
  s = block_sum_256(s, red);
  q = block_sum_256(q, red);
  if (threadIdx.x == 0) { stats[r] = s; stats[rows + r] = q; }
}

// y = (x - mean) * rstd * w + b with mean / rstd from the all-reduced stats over `hidden` = full width
template <typename T>
__global__ void __launch_bounds__(256)
    ln_apply_stats_kernel(const T* __restrict__ x, const float* __restrict__ stats, const T* __restrict__ w,
                          const T* __restrict__ b, T* __restrict__ y, float* __restrict__ mean_out,
                          float* __restrict__ rstd_out, int rows, int cols, float hidden, float eps) {
  const int r = blockIdx.x;
  const float mean = stats[r] / hidden;
  const float var = fmaxf(stats[rows + r] / hidden - mean * mean, 0.f);
  const float rstd = rsqrtf(var + eps);
  if (threadIdx.x == 0) { mean_out[r] = mean; rstd_out[r] = rstd; }
  for (int c = threadIdx.x; c < cols; c += blockDim.x) {
    const float v = (xl_to_float(x[(long long)r * cols + c]) - mean) * rstd;
    y[(long long)r * cols + c] = xl_from_float<T>(v * xl_to_float(w[c]) + xl_to_float(b[c]));
  }
}

XL_API int xl_row_sum_sumsq(const void* x, int dtype, float* stats, int rows, int cols, cudaStream_t s) {
  XL_DISPATCH_DTYPE(dtype, T, { row_sum_sumsq_kernel<T><<<rows, 256, 0, s>>>((const T*)x, stats, rows, cols); });
  return (int)cudaGetLastError();
}
XL_API int xl_ln_apply_stats(const void* x, int dtype, const float* stats, const void* w, const void* b, void* y,
                             float* mean_out, float* rstd_out, int rows, int cols, float hidden, float eps,
                             cudaStream_t s) {
  XL_DISPATCH_DTYPE(dtype, T, {
    ln_apply_stats_kernel<T><<<rows, 256, 0, s>>>((const T*)x, stats, (const T*)w, (const T*)b, (T*)y, mean_out, rstd_out,
                                                 rows, cols, hidden, eps);
  });
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------------------------
// Rows of 16-bit elements -> rows that start on 16-byte boundaries (what TMA needs of a GEMM operand), and back to rows without
// gaps (results with an odd number of columns: the GEMM's own stores of such rows, half a word at every edge of a tile, took
// 1.03 ms for 4096 x 50257 where the padded product and this copy take 0.35 + 0.14 ms). Pure copies, bound by memory: a thread
// moves 16 bytes, read as one or two aligned blocks and shifted together (768 x 50257: 29 us, 5.4 TB/s).
// ------------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    pack_rows_kernel(const uint16_t* __restrict__ src, long long ld_src, uint16_t* __restrict__ dst, long long ld_dst, long long rows,
                     int cols) {
  xl_grid_launch_dependents();
  const int pieces = (int)(ld_dst / 8);
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= pieces) return;
#pragma unroll 4
  for (long long r = blockIdx.y; r < rows; r += gridDim.y) {
    const uint16_t* p = src + r * ld_src + c * 8;
    uint4 o;
    if (c * 8 + 8 <= cols) {
      o = xl_load16_any(p);
    } else {
      uint16_t e[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) e[k] = c * 8 + k < cols ? p[k] : (uint16_t)0;
      o = make_uint4(e[0] | e[1] << 16, e[2] | e[3] << 16, e[4] | e[5] << 16, e[6] | e[7] << 16);
    }
    *reinterpret_cast<uint4*>(dst + r * ld_dst + c * 8) = o;
  }
}
// dst without gaps: a thread writes 8 consecutive elements, which lie in one row or go on in the next ones.
__global__ void __launch_bounds__(256)
    unpack_rows_kernel(const uint16_t* __restrict__ src, long long ld_src, uint16_t* __restrict__ dst, long long rows, unsigned int cols) {
  xl_grid_launch_dependents();
  const long long total = rows * cols;
#pragma unroll 2
  for (long long i = ((long long)blockIdx.x * 256 + threadIdx.x) * 8; i < total; i += (long long)gridDim.x * 256 * 8) {
    long long r = i / cols;
    unsigned int c = (unsigned int)(i - r * cols);
    if (i + 8 <= total && c + 8 <= cols) {
      *reinterpret_cast<uint4*>(dst + i) = xl_load16_any(src + r * ld_src + c);
      continue;
    }
    uint16_t e[8];
    const int n = (int)(total - i < 8 ? total - i : 8);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      e[k] = k < n ? src[r * ld_src + c] : (uint16_t)0;
      if (++c == cols) { c = 0; ++r; }
    }
    if (n == 8) {
      *reinterpret_cast<uint4*>(dst + i) = make_uint4(e[0] | e[1] << 16, e[2] | e[3] << 16, e[4] | e[5] << 16, e[6] | e[7] << 16);
    } else {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < n) dst[i + k] = e[k];
    }
  }
}
// dst (rows, ld_dst) <- src (rows, cols) of 16-bit elements with row stride ld_src, zeros behind; ld_dst a multiple of 8.
XL_API int xl_pack_rows16(const void* src, long long ld_src, void* dst, long long ld_dst, long long rows, int cols, cudaStream_t s) {
  if (rows < 1 || cols < 1 || ld_dst < cols || (ld_dst % 8) || (((uintptr_t)dst) & 15) || (((uintptr_t)src) & 1)) return -1;
  const long long gx = (ld_dst / 8 + 255) / 256;
  long long gy = (16LL * 148 + gx - 1) / gx;
  if (gy > rows) gy = rows;
  pack_rows_kernel<<<dim3((unsigned)gx, (unsigned)gy), 256, 0, s>>>((const uint16_t*)src, ld_src, (uint16_t*)dst, ld_dst, rows, cols);
  return (int)cudaGetLastError();
}
// dst (rows, cols) contiguous <- src (rows, cols) of 16-bit elements with row stride ld_src.
XL_API int xl_unpack_rows16(const void* src, long long ld_src, void* dst, long long rows, int cols, cudaStream_t s) {
  if (rows < 1 || cols < 1 || ld_src < cols || (((uintptr_t)dst) & 15) || (((uintptr_t)src) & 1)) return -1;
  unpack_rows_kernel<<<xl_grid_for(rows * cols, 256 * 8), 256, 0, s>>>((const uint16_t*)src, ld_src, (uint16_t*)dst, rows,
                                                                      (unsigned int)cols);
  return (int)cudaGetLastError();
}
