// What the kernels of the int4 group-quantised product share: codes as 16-bit floats, the MMAs that take them, results.
#pragma once
#include "common.cuh"

#include <math.h>
#include <type_traits>

template <typename T> __device__ __forceinline__ void mma_m16n8k16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  } else {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}

// the first product of a sum: no accumulator registers to clear
template <typename T> __device__ __forceinline__ void mma_m16n8k16_first(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
  } else {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
  }
}
template <typename T> struct GqFmt;
template <> struct GqFmt<__nv_bfloat16> {
  static constexpr uint32_t MASK = 0x000F000Fu, MAGIC = 0x43004300u, ONES = 0x3F803F80u;
  static constexpr float BASE = 128.f;
};
template <> struct GqFmt<__half> {
  static constexpr uint32_t MASK = 0x00F000F0u, MAGIC = 0x54005400u, ONES = 0x3C003C00u;
  static constexpr float BASE = 64.f;
};
// (w & MASK) | MAGIC in one instruction
template <typename T> __device__ __forceinline__ uint32_t gq_place(uint32_t w) {
  uint32_t o;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(o) : "r"(w), "r"(GqFmt<T>::MASK), "r"(GqFmt<T>::MAGIC));
  return o;
}
// w: eight codes, two packed words (the first code of a word in its top nibble). out[i]: codes i and i + 4.
template <typename T> __device__ __forceinline__ void gq_codes8(uint32_t w, uint32_t (&out)[4]) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    out[0] = gq_place<T>(w >> 12);
    out[1] = gq_place<T>(w >> 8);
    out[2] = gq_place<T>(w >> 4);
    out[3] = gq_place<T>(w);
  } else {
    out[0] = gq_place<T>(w >> 8);
    out[1] = gq_place<T>(w >> 4);
    out[2] = gq_place<T>(w);
    out[3] = gq_place<T>(w << 4);
  }
}

struct GqParams {
  const void* x;
  long long ldx;
  const uint16_t* packed;  // (N, K/gs, gs/4), first code of a word in its top nibble
  const void *scale, *zero;  // sz_pairs: scale holds (scale, zero) pairs (K/gs, N, 2); else both (N, K/gs)
  int sz_pairs;
  const void* bias;
  void* y;
  long long ldy;
  int M, N, K, group_size, act_from_col;
  float* slots;            // [grid][2][16 * COLS]
  unsigned int* counters;  // one per tile, zero between launches
  int read_ahead;          // codes, scales and zero points were complete before the previous launch
};

template <typename T> __device__ __forceinline__ T gq_result(const GqParams& p, float sum, float bias, int n) {
  float o = sum + bias;
  if (n >= p.act_from_col) o = 0.5f * o * (1.f + erff(o * 0.70710678118654752f));
  return xl_from_float<T>(o);
}
template <typename T> __device__ __forceinline__ T gq_result(const GqParams& p, float sum, int n) {
  return gq_result<T>(p, sum, p.bias ? xl_to_float(((const T*)p.bias)[n]) : 0.f, n);
}

// Results of a warp that are not finite, from weights that are de-quantised to T first: an infinite activation times a weight is what it
// is elsewhere, and sums overflow only where the products do. The lanes in `mask` have stored row r, channels n .. n + 3; the warp
// takes one result after another. Rare, so it is kept out of the registers of the kernel.
template <typename T, typename S> __device__ __noinline__ void gq_from_weights(const GqParams& p, unsigned mask, int r, int n) {
  const int lane = threadIdx.x & 31, groups = p.K / p.group_size;
  __syncwarp();  // the stored results are read by all lanes
  for (; mask; mask &= mask - 1) {
    const int row = __shfl_sync(0xffffffffu, r, __ffs(mask) - 1), first = __shfl_sync(0xffffffffu, n, __ffs(mask) - 1);
    for (int c = first; c < min(first + 4, p.N); ++c) {
      T* y = (T*)p.y + (long long)row * p.ldy + c;
      if (isfinite(xl_to_float(*y))) continue;
      const uint16_t* codes = p.packed + (long long)c * (p.K / 4);
      float sum = 0.f;
      for (int k = lane * 8; k < p.K; k += 256) {
        const int g = k / p.group_size;
        const S* sz = p.sz_pairs ? (const S*)p.scale + 2 * ((long long)g * p.N + c) : (const S*)p.scale + (long long)c * groups + g;
        const float s = xl_to_float(*sz), z = xl_to_float(p.sz_pairs ? sz[1] : ((const S*)p.zero)[(long long)c * groups + g]);
        float x[8];
        xl_load16((const T*)p.x + (long long)row * p.ldx + k, x);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const float w = xl_to_float(xl_from_float<T>(fmaf((float)((codes[k / 4 + e / 4] >> (12 - 4 * (e & 3))) & 15), s, z)));
          sum = fmaf(x[e], w, sum);
        }
      }
      sum = xl_warp_sum(sum);  // and all lanes have read *y
      if (lane == 0) *y = gq_result<T>(p, sum, c);
    }
  }
}

// gq_gemm_stream.cu. Takes what gq_stream_takes() says; the sizes and pointers are checked by the caller.
bool gq_stream_takes(const GqParams& p);
int gq_stream_launch(const GqParams& p, int ctas, int dtype, int scale_dtype, int* err, cudaStream_t s);
