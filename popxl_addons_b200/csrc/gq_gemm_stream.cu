// int4 group-quantised product of few rows, weights streamed through a ring in shared memory:
//   y[m, n] = sum over blocks b of s[n, b] * (sum_k x[m, k] * q[n, k]) + z[n, b] * (sum_k x[m, k])
// with the arithmetic of gq_codes.cuh (codes on `mma.sync`, scales and zero points on fp32 sums).
//
// Work = (tiles of 128 channels) x (K chunks of 256), tile-major, cut into equal contiguous ranges, one per CTA, one CTA per SM. A CTA
// has a producer (TMA: 16 KB of codes and their scales per chunk, 7 or 8 chunks ahead, which is 130 to 145 KB per SM on its way),
// four warps that bring the tokens' chunk into the order of the MMA fragments together with the sums of x per block, and eight warps that
// multiply: 4 groups of 32 channels x 2 halves of the chunk. The launch's first chunks are on their way while the previous
// kernel still runs, if that does not write them. A tile shared by several CTAs is finished by the one that arrives last; it adds
// the slots of all in CTA order, so results do not depend on timing.
//
// Chains of launches on one B200, us (per-warp double buffers of cp.async in gq_gemm_small_m_kernel -> here):
//             28672 x 4096   4096 x 20480   50400 x 4096   14336 x 2048   2048 x 10240   50400 x 2048   4096 x 1024
//   1 token   29.4 -> 22.5   21.7 -> 18.4   47.9 -> 35.6   11.6 -> 9.9    10.1 -> 8.1    30.5 -> 20.9   8.6 -> 5.2
//   16 tokens 34.8 -> 29.7   27.2 -> 24.1   58.9 -> 47.2   15.1 -> 12.8   13.5 -> 10.7   36.5 -> 28.6   8.5 -> 7.1
// With weights that come from HBM in every launch (three sets in turn), 1 and 16 tokens: 28672 x 4096 31.9 -> 25.2, 40.1 -> 33.3; 14336 x
// 2048 14.8 -> 10.6, 17.7 -> 14.0; 2048 x 10240 12.0 -> 8.3, 16.7 -> 11.4. The ring alone, without the products, takes 13.3 us for 28672 x
// 4096 (5 TB/s). No unit is full (1 and 16 tokens: issue slots 38 and 37 % busy, integer pipe 38 and 32 %, tensor pipe 17 and 26 %, DRAM 29
// and 23 %): what is left is a chunk's chain of wait, loads, eight codes of a word at a time, MMAs and scales in two warps per quarter
// of an SM. Twice as many warps, or codes as subnormal fp16 numbers (20 instead of 28 integer instructions for eight codes, x
// rescaled per chunk), gave 0 to 5 % with up to 8 tokens and lost with more; tcgen05 with the codes as its A operand in TMEM took 33 and
// 42 us for 28672 x 4096 (one block of 64 k values at a time is a chain of hand-overs).
#include "gq_codes.cuh"
#include "tcgen05.cuh"

namespace {

using namespace xl_tc;

constexpr int GS_ROWS = 128, GS_K = 256, GS_BLOCKS = GS_K / 64;
constexpr int GS_MULT = 8, GS_PREP = 4;  // warps
constexpr int GS_THREADS = (GS_MULT + GS_PREP + 1) * 32;
enum { ERR_GS_FULL = 61, ERR_GS_EMPTY = 62, ERR_GS_EMPTY_X = 63 };

template <int NT> struct GsCfg {  // NT: tiles of 8 tokens
  static constexpr int TOK = NT * 8;
  static constexpr int W = GS_ROWS * GS_K / 2, SZ = GS_BLOCKS * GS_ROWS * 4, X = TOK * GS_K * 2, XS = GS_BLOCKS * TOK * 4;
  static constexpr int SZ_AT = W, X_AT = W + SZ, XS_AT = X_AT + X;
  static constexpr int STAGE = (XS_AT + XS + 1023) / 1024 * 1024;
  static constexpr int STAGES = NT == 1 ? 8 : 7;
  static constexpr int RED_LD = GS_ROWS + 4;
  static constexpr int SMEM = STAGES * STAGE + 2 * TOK * RED_LD * 4 + 1024 /*alignment slack*/;
};

__device__ __forceinline__ void gs_mult_sync() { asm volatile("bar.sync 1, %0;" ::"n"(GS_MULT * 32) : "memory"); }

template <typename T, typename S, int NT>
__global__ void __launch_bounds__(GS_THREADS, 1)
    gq_stream_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_sz,
                     const __grid_constant__ GqParams p, int* err) {
  using F = GqFmt<T>;
  using C = GsCfg<NT>;
  constexpr int STAGES = C::STAGES;
  extern __shared__ uint8_t gs_smem[];
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES];
  __shared__ int abort_word;
  __shared__ unsigned int finish;
  uint8_t* ring = (uint8_t*)(((uintptr_t)gs_smem + 1023) & ~(uintptr_t)1023);
  volatile int* abort_flag = &abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, j = lane & 3;
  const int chunks = (p.K + GS_K - 1) / GS_K, n_tiles = (p.N + GS_ROWS - 1) / GS_ROWS, total = n_tiles * chunks;
  const XlRanges ranges{total / (int)gridDim.x, total % (int)gridDim.x};
  const int begin = ranges.begin(blockIdx.x), end = ranges.begin(blockIdx.x + 1);

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 2);  // the producer and the warp that places the tokens
      mbar_init(&empty_bar[s], GS_MULT);
    }
    abort_word = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  if (warp == GS_MULT + GS_PREP) {
    // ------------------------------------------------ weights ------------------------------------------------------
    if (elect_one()) {
      const int per_chunk = p.group_size >= GS_K ? 1 : GS_K / p.group_size;  // groups
      const uint32_t bytes = C::W + per_chunk * GS_ROWS * 4;
      int tile = begin / chunks, ch = begin - tile * chunks;
      auto load = [&](int s) {
        uint8_t* st = ring + s * C::STAGE;
        mbar_expect_tx(&full_bar[s], bytes);
        tma_load_2d(st, &map_w, &full_bar[s], ch * (GS_K / 8), tile * GS_ROWS);
        tma_load_2d(st + C::SZ_AT, &map_sz, &full_bar[s], tile * GS_ROWS, ch * GS_K / p.group_size);
        if (++ch == chunks) { ch = 0; ++tile; }
      };
      const int items = end - begin, ahead = min(STAGES, items);
      if (!p.read_ahead) xl_grid_dependency_wait();
      for (int i = 0; i < ahead; ++i) load(i);
      xl_grid_dependency_wait();  // no bounded wait runs while the previous kernel still does
      int stage = 0;
      uint32_t phase = 0;
      for (int i = ahead; i < items; ++i) {
        if (!mbar_wait(&empty_bar[stage], phase, abort_flag, err, ERR_GS_EMPTY)) break;
        load(stage);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (*abort_flag)
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);  // copies in flight arrive before the CTA gives its memory back
    }
    return;
  }
  xl_grid_dependency_wait();
  xl_grid_launch_dependents();

  if (warp >= GS_MULT) {
    // ------------------------------------------------ tokens -------------------------------------------------------
    const T* x = (const T*)p.x;
    const int items = end - begin;
    for (int i = warp - GS_MULT; i < items; i += GS_PREP) {
      const int ch = (begin + i) % chunks, stage = i % STAGES;
      uint4 v[GS_BLOCKS][NT][2];
#pragma unroll
      for (int b = 0; b < GS_BLOCKS; ++b)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int k = ch * GS_K + b * 64 + (j * 2 + q) * 8, tok = t * 8 + g;
            v[b][t][q] = tok < p.M && k < p.K ? *reinterpret_cast<const uint4*>(x + tok * p.ldx + k) : make_uint4(0, 0, 0, 0);
          }
      if (i >= STAGES && !mbar_wait_warp(&empty_bar[stage], (i / STAGES - 1) & 1, abort_flag, err, ERR_GS_EMPTY_X)) break;
      uint4* xf = reinterpret_cast<uint4*>(ring + stage * C::STAGE + C::X_AT);
      float* xs = reinterpret_cast<float*>(ring + stage * C::STAGE + C::XS_AT);
      const uint32_t ones[4] = {F::ONES, F::ONES, F::ONES, F::ONES};
#pragma unroll
      for (int b = 0; b < GS_BLOCKS; ++b)
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          float sum[4];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const uint4 r = v[b][t][q];  // to the order of the codes: (0, 4), (1, 5), (2, 6), (3, 7)
            const uint4 f = make_uint4(__byte_perm(r.x, r.z, 0x5410), __byte_perm(r.x, r.z, 0x7632), __byte_perm(r.y, r.w, 0x5410),
                                       __byte_perm(r.y, r.w, 0x7632));
            xf[((b * NT + t) * 2 + q) * 32 + lane] = f;
            if (q == 0) mma_m16n8k16_first<T>(sum, ones, f.x, f.y);
            else mma_m16n8k16<T>(sum, ones, f.x, f.y);
            mma_m16n8k16<T>(sum, ones, f.z, f.w);
          }
          if (lane < 4) *reinterpret_cast<float2*>(xs + b * C::TOK + t * 8 + 2 * lane) = make_float2(sum[0], sum[1]);
        }
      __syncwarp();
      if (lane == 0) mbar_arrive(&full_bar[stage]);
    }
    return;
  }

  // ---------------------------------------------------- products ---------------------------------------------------
  float* red = reinterpret_cast<float*>(ring + STAGES * C::STAGE);
  const int rows0 = (warp & 3) * 32, half = warp >> 2;  // 32 channels x blocks 2 * half, 2 * half + 1 of every chunk
  // Row g of an MMA tile is channel `perm`: the four rows of a half-warp are 2 apart, so that the swizzled 32-byte pieces they read
  // lie in different banks.
  const int perm = 2 * (g & 3) + (g >> 2);
  const int shift = p.group_size == 64 ? 0 : (p.group_size == 128 ? 1 : 2);
  int code_at[2], sz_at[2];
#pragma unroll
  for (int b = 0; b < 2; ++b) {
    const int blk = half * 2 + b;
    code_at[b] = (rows0 + perm) * 128 + ((2 * blk + (j >> 1)) ^ perm) * 16 + (j & 1) * 8;
    sz_at[b] = C::SZ_AT + ((blk >> shift) * GS_ROWS + rows0 + perm) * 4;
  }
  const int x_at = C::X_AT + (half * 2 * NT * 2 * 32 + lane) * 16, xs_at = C::XS_AT + (half * 2 * C::TOK + 2 * j) * 4;
  int stage = 0;
  uint32_t phase = 0;
  bool ok = true;  // a warp that gave up still meets the others at the barriers
  const int first_tile = begin / chunks;
  for (int item = begin; item < end;) {
    const int tile = item / chunks, n_base = tile * GS_ROWS, c0 = item - tile * chunks, c1 = min(chunks, c0 + (end - item));
    float acc[2][NT][4], bias[4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][t][e] = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e)  // of the channels whose results this lane stores, long before
      bias[e] = p.bias && n_base + lane * 4 + e < p.N ? xl_to_float(((const T*)p.bias)[n_base + lane * 4 + e]) : 0.f;
    for (int c = c0; c < c1 && ok; ++c) {
      ok = mbar_wait_warp(&full_bar[stage], phase, abort_flag, err, ERR_GS_FULL);
      if (!ok) break;
      const uint8_t* st = ring + stage * C::STAGE;
#pragma unroll
      for (int b = 0; b < 2; ++b) {
        uint4 xb[NT][2];
        float2 xs[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) {
#pragma unroll
          for (int q = 0; q < 2; ++q) xb[t][q] = *reinterpret_cast<const uint4*>(st + x_at + ((b * NT + t) * 2 + q) * 512);
          xs[t] = *reinterpret_cast<const float2*>(st + xs_at + (b * C::TOK + t * 8) * 4);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const uint2 lo = *reinterpret_cast<const uint2*>(st + code_at[b] + i * 2048);
          const uint2 hi = *reinterpret_cast<const uint2*>(st + code_at[b] + i * 2048 + 1024);
          const uint32_t sz_lo = *reinterpret_cast<const uint32_t*>(st + sz_at[b] + i * 64);
          const uint32_t sz_hi = *reinterpret_cast<const uint32_t*>(st + sz_at[b] + i * 64 + 32);
          float part[NT][4];
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            uint32_t cl[4], chh[4];
            gq_codes8<T>(q ? lo.y : lo.x, cl);
            gq_codes8<T>(q ? hi.y : hi.x, chh);
            const uint32_t a0[4] = {cl[0], chh[0], cl[1], chh[1]}, a1[4] = {cl[2], chh[2], cl[3], chh[3]};
#pragma unroll
            for (int t = 0; t < NT; ++t) {
              if (q == 0) mma_m16n8k16_first<T>(part[t], a0, xb[t][0].x, xb[t][0].y);
              else mma_m16n8k16<T>(part[t], a0, xb[t][1].x, xb[t][1].y);
            }
#pragma unroll
            for (int t = 0; t < NT; ++t) mma_m16n8k16<T>(part[t], a1, xb[t][q].z, xb[t][q].w);
          }
          const float2 wl = xl_pair_to_float2<S>(sz_lo), wh = xl_pair_to_float2<S>(sz_hi);
          const float zl = fmaf(-F::BASE, wl.x, wl.y), zh = fmaf(-F::BASE, wh.x, wh.y);
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            acc[i][t][0] = fmaf(wl.x, part[t][0], fmaf(zl, xs[t].x, acc[i][t][0]));
            acc[i][t][1] = fmaf(wl.x, part[t][1], fmaf(zl, xs[t].y, acc[i][t][1]));
            acc[i][t][2] = fmaf(wh.x, part[t][2], fmaf(zh, xs[t].x, acc[i][t][2]));
            acc[i][t][3] = fmaf(wh.x, part[t][3], fmaf(zh, xs[t].y, acc[i][t][3]));
          }
        }
      }
      mbar_arrive_reads_done(&empty_bar[stage]);
      if (++stage == STAGES) { stage = 0; phase ^= 1; }
    }
    // the two halves of K meet in shared memory
    gs_mult_sync();  // readers of the previous segment are done with `red`
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          red[(half * C::TOK + t * 8 + 2 * j + (e & 1)) * C::RED_LD + rows0 + i * 16 + perm + (e >> 1) * 8] = acc[i][t][e];
    gs_mult_sync();
    auto together = [&](int r, int col) {
      float4 v = *reinterpret_cast<const float4*>(red + r * C::RED_LD + col);
      const float4 o = *reinterpret_cast<const float4*>(red + (C::TOK + r) * C::RED_LD + col);
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
      return v;
    };
    const bool whole = c1 - c0 == chunks;
    bool finishing = whole;
    if (!whole) {
      float* slot = p.slots + ((long long)blockIdx.x * 2 + (tile == first_tile ? 0 : 1)) * (16 * GS_ROWS);
      for (int i = threadIdx.x; i < p.M * (GS_ROWS / 4); i += GS_MULT * 32) {
        const int r = i / (GS_ROWS / 4), col = i % (GS_ROWS / 4) * 4;
        __stcg(reinterpret_cast<float4*>(slot + r * GS_ROWS + col), together(r, col));
      }
      gs_mult_sync();
      if (threadIdx.x == 0) {
        __threadfence();  // for the stores of all, which the barrier has ordered before it
        finish = atomicAdd(p.counters + tile, (unsigned int)(c1 - c0)) + (unsigned int)(c1 - c0) == (unsigned int)chunks;
      }
      gs_mult_sync();
      finishing = finish != 0;
      if (finishing) __threadfence();
    }
    if (finishing) {
      // CTAs that share the tile, in order: all but the first begin inside it (slot 0), the first may hold an earlier tile too
      int cta0 = blockIdx.x, cta1 = blockIdx.x, slot0 = 0;
      if (!whole) {
        cta0 = ranges.owner(tile * chunks);
        cta1 = ranges.owner(tile * chunks + chunks - 1);
        slot0 = ranges.begin(cta0) < tile * chunks ? 1 : 0;
      }
      for (int r = warp; r < p.M; r += GS_MULT) {  // a warp: 128 channels of a token
        const int col = lane * 4, n = n_base + col;
        const bool on = n < p.N;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (on && whole) {
          v = together(r, col);
        } else if (on) {
          const float* base = p.slots + r * GS_ROWS + col;
#pragma unroll 8
          for (int k = cta0; k <= cta1; ++k) {
            const float4 o = __ldcg(reinterpret_cast<const float4*>(base + ((long long)k * 2 + (k == cta0 ? slot0 : 0)) * (16 * GS_ROWS)));
            v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
          }
        }
        const float o[4] = {v.x, v.y, v.z, v.w};
        T* yr = (T*)p.y + (long long)r * p.ldy + n;
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (on && n + e < p.N) yr[e] = gq_result<T>(p, o[e], bias[e], n + e);
        const unsigned bad = __ballot_sync(0xffffffffu, on && !(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w)));
        if (bad) gq_from_weights<T, S>(p, bad, r, n);
      }
      if (!whole && threadIdx.x == 0) p.counters[tile] = 0;
    }
    item += c1 - c0;
  }
}

// 2-D map of 32-bit words, `rows` of `cols` (a multiple of 4)
int gs_map(CUtensorMap* map, const void* ptr, long long cols, long long rows, int box_cols, int box_rows, CUtensorMapSwizzle swizzle) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return (int)cudaErrorNotSupported;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)cols * 4};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, (void*)ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : (int)cudaErrorInvalidValue;
}

template <typename T, typename S, int NT> int gs_launch(const GqParams& p, int ctas, int* err, cudaStream_t s) {
  using C = GsCfg<NT>;
  static XlPerDevice smem;
  XL_TRY(xl_allow_smem(gq_stream_kernel<T, S, NT>, C::SMEM, smem));
  const long long total = (long long)((p.N + GS_ROWS - 1) / GS_ROWS) * ((p.K + GS_K - 1) / GS_K);
  if (total > (1 << 30)) return -1;
  CUtensorMap mw, msz;
  int rc = gs_map(&mw, p.packed, p.K / 8, p.N, GS_K / 8, GS_ROWS, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc == 0)
    rc = gs_map(&msz, p.scale, p.N, p.K / p.group_size, GS_ROWS, p.group_size >= GS_K ? 1 : GS_K / p.group_size, CU_TENSOR_MAP_SWIZZLE_NONE);
  if (rc) return rc;
  const cudaError_t e = xl_launch_overlapped(gq_stream_kernel<T, S, NT>, dim3((unsigned)(total < ctas ? total : ctas)), dim3(GS_THREADS),
                                             (size_t)C::SMEM, s, mw, msz, p, err);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}
template <typename T, typename S> int gs_pick(const GqParams& p, int ctas, int* err, cudaStream_t s) {
  return p.M <= 8 ? gs_launch<T, S, 1>(p, ctas, err, s) : gs_launch<T, S, 2>(p, ctas, err, s);
}

}  // namespace

// Scales and zero points as pairs, rows of pairs of whole 16-byte pieces; a chunk of K holds whole groups or lies in one.
XL_API int xl_gq_gemm_streams(int N, int group_size, int sz_pairs) {
  return sz_pairs && N % 4 == 0 && (group_size % GS_K == 0 || group_size == 64 || group_size == 128);
}
bool gq_stream_takes(const GqParams& p) { return xl_gq_gemm_streams(p.N, p.group_size, p.sz_pairs); }

int gq_stream_launch(const GqParams& p, int ctas, int dtype, int scale_dtype, int* err, cudaStream_t s) {
  if (dtype == XL_BF16)
    return scale_dtype == XL_F16 ? gs_pick<__nv_bfloat16, __half>(p, ctas, err, s) : gs_pick<__nv_bfloat16, __nv_bfloat16>(p, ctas, err, s);
  return scale_dtype == XL_F16 ? gs_pick<__half, __half>(p, ctas, err, s) : gs_pick<__half, __nv_bfloat16>(p, ctas, err, s);
}
