// Kernels of the token-by-token decoding path (batch of a few sequences, one new token each):
//   xl_gq_gemm_small_m   y[M<=16, N] = x[M, K] * dequant(Wq)[K, N] (+ bias): 4-bit group-quantised weights are streamed
//                        once and fed to the tensor cores as codes; scales and zero points meet the fp32 sums
//   xl_rotary_at         rotary embedding of the new tokens at a position read from device memory
//   xl_kv_append         write the new keys / values into the KV cache at that position
//   xl_argmax_rows       greedy sampling: per-row (max, index) of the local logits slice
// Everything that depends on the current position reads it from a device word, so one decoding step has no
// launch-time argument that changes between steps and can be replayed as a CUDA graph.
//
// The int4 GEMM is bandwidth-bound by construction (M <= 16), so it uses the register-operand `mma.sync.m16n8k16` form: its
// operands come straight from the registers that hold the freshly unpacked codes, which is exactly what a streaming kernel wants.
// (tcgen05 needs its operands in shared memory or TMEM; for prefill-sized M the weights are de-quantised once and the tcgen05 GEMM
// is used.)
#include "common.cuh"
#include "gq_codes.cuh"

#include <cooperative_groups.h>

// ------------------------------------------------------------------------------------------------------------------
// int4 group-quantised GEMM, M <= 16
// ------------------------------------------------------------------------------------------------------------------
// y[m, n] = sum over blocks b of s[n, b] * (sum_k x[m, k] * q[n, k]) + z[n, b] * (sum_k x[m, k]), q the 4-bit codes: scale and zero
// point are applied to fp32 sums, so the weights themselves are never rounded to 16 bits, and a code costs less than one
// instruction: a nibble moved into the mantissa of a 16-bit float with a suitable exponent IS the number BASE + n (bf16:
// 0x4300 | n = 128 + n; fp16: 0x5400 | n << 4 = 64 + n), two at a time, and the base goes with the zero point.
// (De-quantising every weight to 16 bits took 5.5 instructions per weight, 46 % of the issue slots at a fifth of the bandwidth.
// Both halves of the sum are of the size of BASE * |x|: activations above 2^120 overflow, and an infinite one gives NaN. Results that
// are not finite are therefore taken again from the weights themselves, gq_from_weights.)
//
// The channels are the rows of the `mma.sync.m16n8k16` tiles and the tokens their columns, so up to 8 tokens take one MMA per 256
// weights and 9 to 16 tokens two. Lane (quad g, j) holds rows g and g + 8; of every block of 64 (or 32) k values lane j of a quad
// feeds 16 (8) consecutive ones. Any assignment of k values to the k slots of an MMA is valid as long as both operands agree: the
// codes k and k + 4 of eight consecutive ones lie 16 bits apart, so x is permuted to (0, 4), (1, 5), ... once per chunk. An MMA
// whose weights are all ones gives the sums of x in the layout of the accumulators.
//
// Work = (tiles of CT * 16 channels) x (K chunks of 128), tile-major, cut into equal contiguous ranges, one per CTA (one CTA per
// SM): the grid is sized to the machine, not to the problem. Warps take the chunks of a tile segment in turn; weights, scales and
// zero points reach them through per-warp double buffers filled with cp.async. A tile shared by several CTAs is finished by the one
// that arrives last: every CTA leaves its sums in a slot of its own and the finisher adds the slots in CTA order, so results do
// not depend on timing. A launch requests its first weights while its predecessor drains, if that does not write them.
constexpr int GQ_KCHUNK = 128;

// NT: tiles of 8 tokens; WPB: 32-bit words of codes per lane and block (2: blocks of 64 k values, 1: of 32)
template <int NT, int WPB> struct GqCfg {
  static constexpr int WARPS = NT == 1 ? 16 : 8;  // as many as the registers allow
  static constexpr int CT = NT == 1 ? 4 : 8;      // with more tokens wider tiles, so that x is read less often
  static constexpr int COLS = CT * 16;
  static constexpr int BLOCKS = GQ_KCHUNK / (32 * WPB);
  static constexpr int CODE_UNITS = CT * 64;                 // 16-byte units of codes per stage
  static constexpr int SZ_UNITS = BLOCKS * COLS / 4;         // (scale, zero) pairs of 16-bit numbers, four channels per unit
  static constexpr int STAGE_UNITS = CODE_UNITS + SZ_UNITS;
  static constexpr int RED_LD = COLS + 4;
  static constexpr int RED_FLOATS = WARPS * NT * 8 * RED_LD;
  static constexpr int SMEM = WARPS * 2 * STAGE_UNITS * 16 + RED_FLOATS * 4;
};

template <typename T, typename S, int NT, int WPB>
__global__ void __launch_bounds__(GqCfg<NT, WPB>::WARPS * 32, 1)
    gq_gemm_small_m_kernel(const __grid_constant__ GqParams p) {
  using F = GqFmt<T>;
  using C = GqCfg<NT, WPB>;
  constexpr int CT = C::CT, COLS = C::COLS, BLOCKS = C::BLOCKS, SB = 32 * WPB, WARPS = C::WARPS;
  extern __shared__ uint4 gq_smem[];
  __shared__ unsigned int finish;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, j = lane & 3;
  uint4* ring = gq_smem + warp * (2 * C::STAGE_UNITS);
  float* red = reinterpret_cast<float*>(gq_smem + WARPS * 2 * C::STAGE_UNITS);
  const int chunks = p.K / GQ_KCHUNK, n_tiles = (p.N + COLS - 1) / COLS, groups = p.K / p.group_size;
  const int total = n_tiles * chunks;
  const XlRanges ranges{total / (int)gridDim.x, total % (int)gridDim.x};
  int item = ranges.begin(blockIdx.x);
  const int item_end = ranges.begin(blockIdx.x + 1);
  const int first_tile = item / chunks;
  const bool pairs16 = p.sz_pairs && p.N % 4 == 0;  // scales and zero points can be copied 16 bytes at a time
  const T* x = (const T*)p.x;

  // The chunks of this warp over the whole range, tile after tile. What a request needs of a tile is worked out once per tile: this
  // lane's first row of codes, which of its rows exist, and its first unit of scales and zero points.
  struct Cursor { int item, c1, ch, tile; };  // first item of the current tile segment, its end chunk, current chunk, tile
  const int bpg = p.group_size / SB;          // blocks per group
  const long long row_step = 8LL * (p.K / 4);
  const int sz_b = lane / (COLS / 4), sz_n = (lane % (COLS / 4)) * 4;  // unit `lane`; unit 32 i + lane lies i * SZ_STEP blocks on
  constexpr int SZ_STEP = 32 / (COLS / 4);
  auto segment = [&](Cursor& c) {
    while (c.item < item_end) {
      c.tile = c.item / chunks;
      const int c0 = c.item - c.tile * chunks;
      c.c1 = min(chunks, c0 + (item_end - c.item));
      c.ch = c0 + warp;
      if (c.ch < c.c1) return;
      c.item += c.c1 - c0;
    }
  };
  auto advance = [&](Cursor& c) -> bool {  // whether the tile changed
    if (c.item >= item_end) return false;
    c.ch += WARPS;
    if (c.ch < c.c1) return false;
    c.item = c.tile * chunks + c.c1;
    segment(c);
    return true;
  };
  const uint16_t* row0 = p.packed;  // of the tile that is requested next
  int rows_on = 0;                  // its rows 8 i + g below N
  auto enter = [&](const Cursor& c) {
    if (c.item >= item_end) return;
    const int n = c.tile * COLS + g;
    row0 = p.packed + (long long)n * (p.K / 4) + j * 8;
    rows_on = (p.N - n + 7) / 8;
  };
  // Codes of a tile of 16 channels: piece q (32 codes) of row r at unit q * 16 + (r ^ 4 * (q & 1)), so that the eight-byte reads
  // below touch every bank once.
  uint4* const code_dst = ring + j * 16 + (g ^ ((j & 1) * 4));
  auto request = [&](const Cursor& c, int buf) {
    if (c.item < item_end) {
      uint4* dst = code_dst + buf * C::STAGE_UNITS;
      const uint16_t* src = row0 + c.ch * (GQ_KCHUNK / 4);
#pragma unroll
      for (int i = 0; i < CT * 2; ++i) {
        const bool on = i < rows_on;
        xl_cp_async16(dst + (i >> 1) * 64 + (i & 1) * 8, on ? src : p.packed, on);
        src += row_step;
      }
      uint4* sz = ring + buf * C::STAGE_UNITS + C::CODE_UNITS;
      const int n = c.tile * COLS + sz_n;
#pragma unroll
      for (int i = 0; i < (C::SZ_UNITS + 31) / 32; ++i) {
        const int u = i * 32 + lane, block = c.ch * BLOCKS + sz_b + i * SZ_STEP;
        const int grp = bpg == 1 ? block : block / bpg;
        if (C::SZ_UNITS % 32 == 0 || u < C::SZ_UNITS) {
          if (pairs16) {
            const bool on = n < p.N;
            xl_cp_async16(sz + u, (const uint32_t*)p.scale + (on ? (long long)grp * p.N + n : 0), on);
          } else {
            uint32_t v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              v[e] = 0;
              if (n + e < p.N) {
                if (p.sz_pairs) {
                  v[e] = ((const uint32_t*)p.scale)[(long long)grp * p.N + n + e];
                } else {
                  const long long at = (long long)(n + e) * groups + grp;
                  v[e] = ((const uint16_t*)p.scale)[at] | ((uint32_t)((const uint16_t*)p.zero)[at] << 16);
                }
              }
            }
            sz[u] = make_uint4(v[0], v[1], v[2], v[3]);
          }
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");  // possibly empty: one group per chunk slot
  };
  auto load_x = [&](const Cursor& c, int b, uint4 (&v)[NT][WPB]) {
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int q = 0; q < WPB; ++q)
        v[t][q] = c.item < item_end && t * 8 + g < p.M
                      ? *reinterpret_cast<const uint4*>(x + (t * 8 + g) * p.ldx + c.ch * GQ_KCHUNK + b * SB + (j * WPB + q) * 8)
                      : make_uint4(0, 0, 0, 0);
  };

  Cursor ahead{item, 0, 0, 0};
  segment(ahead);
  Cursor cur = ahead;
  enter(ahead);
  if (!p.read_ahead) xl_grid_dependency_wait();
  request(ahead, 0);
  if (advance(ahead)) enter(ahead);
  request(ahead, 1);
  if (advance(ahead)) enter(ahead);
  xl_grid_dependency_wait();  // the first weights are on their way; everything else may come from the previous kernel
  xl_grid_launch_dependents();
  uint4 xn[NT][WPB];
  load_x(cur, 0, xn);
  int buf = 0;
  while (item < item_end) {
    const int tile = item / chunks, n_base = tile * COLS;
    const int c0 = item - tile * chunks;
    const int c1 = min(chunks, c0 + (item_end - item));
    float acc[CT][NT][4];
#pragma unroll
    for (int i = 0; i < CT; ++i)
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][t][e] = 0.f;
    for (int ch = c0 + warp; ch < c1; ch += WARPS) {
      Cursor next = cur;
      advance(next);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();  // lanes read pieces that other lanes of the warp copied
      const uint32_t* codes = reinterpret_cast<const uint32_t*>(ring + buf * C::STAGE_UNITS);
      const uint32_t* sz = codes + C::CODE_UNITS * 4;
#pragma unroll
      for (int b = 0; b < BLOCKS; ++b) {
        uint32_t xb[NT][WPB][4];  // the B operand: x of codes (0, 4), (1, 5), (2, 6), (3, 7)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
          for (int q = 0; q < WPB; ++q) {
            const uint4 v = xn[t][q];
            xb[t][q][0] = __byte_perm(v.x, v.z, 0x5410);
            xb[t][q][1] = __byte_perm(v.x, v.z, 0x7632);
            xb[t][q][2] = __byte_perm(v.y, v.w, 0x5410);
            xb[t][q][3] = __byte_perm(v.y, v.w, 0x7632);
          }
        load_x(b + 1 < BLOCKS ? cur : next, b + 1 < BLOCKS ? b + 1 : 0, xn);  // one block ahead
        float xs[NT][4];  // [0], [1]: sums of x of tokens 2j, 2j + 1
#pragma unroll
        for (int t = 0; t < NT; ++t) {
          const uint32_t ones[4] = {F::ONES, F::ONES, F::ONES, F::ONES};
#pragma unroll
          for (int q = 0; q < WPB; ++q) {
            if (q == 0) mma_m16n8k16_first<T>(xs[t], ones, xb[t][q][0], xb[t][q][1]);
            else mma_m16n8k16<T>(xs[t], ones, xb[t][q][0], xb[t][q][1]);
            mma_m16n8k16<T>(xs[t], ones, xb[t][q][2], xb[t][q][3]);
          }
        }
#pragma unroll
        for (int i = 0; i < CT; ++i) {
          uint32_t lo[WPB], hi[WPB];  // rows g and g + 8
          if constexpr (WPB == 2) {
            const int piece = b * 2 + (j >> 1), sw = (piece & 1) * 4;
            const uint2 a = *reinterpret_cast<const uint2*>(codes + (i * 64 + piece * 16 + (g ^ sw)) * 4 + (j & 1) * 2);
            const uint2 c = *reinterpret_cast<const uint2*>(codes + (i * 64 + piece * 16 + ((g + 8) ^ sw)) * 4 + (j & 1) * 2);
            lo[0] = a.x; lo[1] = a.y; hi[0] = c.x; hi[1] = c.y;
          } else {
            const int sw = (b & 1) * 4;
            lo[0] = codes[(i * 64 + b * 16 + (g ^ sw)) * 4 + j];
            hi[0] = codes[(i * 64 + b * 16 + ((g + 8) ^ sw)) * 4 + j];
          }
          const uint32_t sz_lo = sz[b * COLS + i * 16 + g], sz_hi = sz[b * COLS + i * 16 + g + 8];
          float part[NT][4];
#pragma unroll
          for (int q = 0; q < WPB; ++q) {
            uint32_t cl[4], chh[4];
            gq_codes8<T>(lo[q], cl);
            gq_codes8<T>(hi[q], chh);
            const uint32_t a0[4] = {cl[0], chh[0], cl[1], chh[1]}, a1[4] = {cl[2], chh[2], cl[3], chh[3]};
#pragma unroll
            for (int t = 0; t < NT; ++t) {
              if (q == 0) mma_m16n8k16_first<T>(part[t], a0, xb[t][q][0], xb[t][q][1]);
              else mma_m16n8k16<T>(part[t], a0, xb[t][q][0], xb[t][q][1]);
              mma_m16n8k16<T>(part[t], a1, xb[t][q][2], xb[t][q][3]);
            }
          }
          const float2 wl = xl_pair_to_float2<S>(sz_lo), wh = xl_pair_to_float2<S>(sz_hi);
          const float zl = fmaf(-F::BASE, wl.x, wl.y), zh = fmaf(-F::BASE, wh.x, wh.y);
#pragma unroll
          for (int t = 0; t < NT; ++t) {
            acc[i][t][0] = fmaf(wl.x, part[t][0], fmaf(zl, xs[t][0], acc[i][t][0]));
            acc[i][t][1] = fmaf(wl.x, part[t][1], fmaf(zl, xs[t][1], acc[i][t][1]));
            acc[i][t][2] = fmaf(wh.x, part[t][2], fmaf(zh, xs[t][0], acc[i][t][2]));
            acc[i][t][3] = fmaf(wh.x, part[t][3], fmaf(zh, xs[t][1], acc[i][t][3]));
          }
        }
      }
      __syncwarp();  // all lanes have read this stage
      request(ahead, buf);
      if (advance(ahead)) enter(ahead);
      cur = next;
      buf ^= 1;
    }
    // add the K slices of the warps up in shared memory
    __syncthreads();  // readers of the previous segment are done with `red`
#pragma unroll
    for (int i = 0; i < CT; ++i)
#pragma unroll
      for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          red[(warp * NT * 8 + t * 8 + 2 * j + (e & 1)) * C::RED_LD + i * 16 + g + (e >> 1) * 8] = acc[i][t][e];
    __syncthreads();
    const bool whole = c1 - c0 == chunks;
    bool finishing = whole;
    if (!whole) {
      float* slot = p.slots + ((long long)blockIdx.x * 2 + (tile == first_tile ? 0 : 1)) * (16 * COLS);
      for (int i = threadIdx.x; i < p.M * (COLS / 4); i += blockDim.x) {
        const int r = i / (COLS / 4), col = i % (COLS / 4) * 4;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
          const float4 o = *reinterpret_cast<const float4*>(red + (w * NT * 8 + r) * C::RED_LD + col);
          s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
        }
        __stcg(reinterpret_cast<float4*>(slot + r * COLS + col), s);
      }
      __threadfence();
      __syncthreads();
      if (threadIdx.x == 0)
        finish = atomicAdd(p.counters + tile, (unsigned int)(c1 - c0)) + (unsigned int)(c1 - c0) == (unsigned int)chunks;
      __syncthreads();
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
      for (int i0 = warp * 32; i0 < p.M * (COLS / 4); i0 += WARPS * 32) {  // whole warps
        const int i = i0 + lane, r = i / (COLS / 4), col = i % (COLS / 4) * 4, n = n_base + col;
        const bool on = r < p.M && n < p.N;
        float v[4] = {0.f, 0.f, 0.f, 0.f};
        if (on && whole) {
#pragma unroll
          for (int w = 0; w < WARPS; ++w) {
            const float4 o = *reinterpret_cast<const float4*>(red + (w * NT * 8 + r) * C::RED_LD + col);
            v[0] += o.x; v[1] += o.y; v[2] += o.z; v[3] += o.w;
          }
        } else if (on) {
          const float* base = p.slots + r * COLS + col;
#pragma unroll 4
          for (int k = cta0; k <= cta1; ++k) {
            const float4 o = __ldcg(reinterpret_cast<const float4*>(base + ((long long)k * 2 + (k == cta0 ? slot0 : 0)) * (16 * COLS)));
            v[0] += o.x; v[1] += o.y; v[2] += o.z; v[3] += o.w;
          }
        }
        T* yr = (T*)p.y + (long long)r * p.ldy + n;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (on && n + e < p.N) yr[e] = gq_result<T>(p, v[e], n + e);
        }
        // (a channel from N on has zero codes, scale and zero point: 0, or NaN for nothing that is stored)
        const unsigned bad = __ballot_sync(0xffffffffu, on && !(isfinite(v[0]) && isfinite(v[1]) && isfinite(v[2]) && isfinite(v[3])));
        if (bad) gq_from_weights<T, S>(p, bad, r, n);
      }
      if (!whole && threadIdx.x == 0) p.counters[tile] = 0;
    }
    item += c1 - c0;
  }
}

template <typename T, typename S, int NT, int WPB> static int gq_small_launch(const GqParams& p, int ctas, cudaStream_t s) {
  using C = GqCfg<NT, WPB>;
  static XlPerDevice smem;
  XL_TRY(xl_allow_smem(gq_gemm_small_m_kernel<T, S, NT, WPB>, C::SMEM, smem));
  const long long total = (long long)((p.N + C::COLS - 1) / C::COLS) * (p.K / GQ_KCHUNK);
  if (total > (1 << 30)) return -1;
  const int grid = (int)(total < ctas ? total : ctas);
  const cudaError_t e = xl_launch_overlapped(gq_gemm_small_m_kernel<T, S, NT, WPB>, dim3((unsigned)grid), dim3(C::WARPS * 32),
                                             (size_t)C::SMEM, s, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}
template <typename T, typename S> static int gq_small_pick(const GqParams& p, int ctas, cudaStream_t s) {
  // a scale per 64 k values and more: blocks of 64, half as many scales to apply; up to 8 tokens: half the MMAs
  if (p.group_size % 64 == 0)
    return p.M <= 8 ? gq_small_launch<T, S, 1, 2>(p, ctas, s) : gq_small_launch<T, S, 2, 2>(p, ctas, s);
  return p.M <= 8 ? gq_small_launch<T, S, 1, 1>(p, ctas, s) : gq_small_launch<T, S, 2, 1>(p, ctas, s);
}

// Floats of `slots` for a grid of `ctas`; `counters` needs ceil(N / 64) zero-initialised words (left zeroed).
XL_API int xl_gq_gemm_small_m_slots(int ctas) { return ctas * 2 * 16 * 128; }

// Scales as pairs with groups of 64, 128 or a multiple of 256 go through the ring of gq_gemm_stream.cu (figures there), everything else
// through the kernel above. `err`: error word of its waits.
// Requirements: M <= 16, K % 128 == 0, group_size % 32 == 0, 16-byte aligned x rows and weight rows. `ctas`: size of the grid (one
// per SM). sz_pairs: `scale` holds (scale, zero) pairs laid out (K/gs, N, 2) and `zero` is unused. act_from_col: first column that
// gets GELU (>= N: none). `dtype`: type of x, bias and y (fp16 or bf16); `scale_dtype`: type of the per-group scale and zero
// point (fp16 / bf16). read_ahead: packed, scale and zero were complete before the previous launch on the stream. Returns -1 for
// unsupported arguments.
XL_API int xl_gq_gemm_small_m(const void* x, const void* packed, const void* scale, const void* zero, const void* bias,
                              void* y, int M, int N, int K, int group_size, long long ldx, long long ldy, int act_from_col,
                              int ctas, float* slots, unsigned int* counters, int dtype, int scale_dtype, int sz_pairs,
                              int read_ahead, int* err, cudaStream_t s) {
  if (M < 1 || M > 16 || N < 1 || K < GQ_KCHUNK || K % GQ_KCHUNK || group_size < 32 || group_size % 32 || K % group_size ||
      dtype == XL_F32 || scale_dtype == XL_F32)
    return -1;
  if ((ldx % 8) || ctas < 1 || !slots || !counters || (((uintptr_t)x | (uintptr_t)packed | (uintptr_t)scale) & 15)) return -1;
  const GqParams p{x, ldx, (const uint16_t*)packed, scale, zero, sz_pairs, bias, y, ldy, M, N, K, group_size, act_from_col, slots,
                   counters, read_ahead};
  if (gq_stream_takes(p)) return gq_stream_launch(p, ctas, dtype, scale_dtype, err, s);
  if (dtype == XL_BF16)
    return scale_dtype == XL_F16 ? gq_small_pick<__nv_bfloat16, __half>(p, ctas, s) : gq_small_pick<__nv_bfloat16, __nv_bfloat16>(p, ctas, s);
  return scale_dtype == XL_F16 ? gq_small_pick<__half, __half>(p, ctas, s) : gq_small_pick<__half, __nv_bfloat16>(p, ctas, s);
}

// ------------------------------------------------------------------------------------------------------------------
// Rotary at a device-side position + KV-cache append, one launch.
// qkv: rows of `ld` elements whose first 3*H*D hold the new-token projections [q | k | v]; rotates q and k in place
// (first R features of each head, interleaved pairs) for position pos = *pos_ptr and writes k, v into the caches
// (B, H, Smax, D) at that position. sin / cos tables: (Smax, R/2). One thread per (b, h, feature pair).
// ------------------------------------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
    rotary_append_kernel(T* qkv, long long ld, const T* sin_t, const T* cos_t, T* k_cache, T* v_cache,
                         const int* pos_ptr, int B, int H, int D, int R, int Smax) {
  xl_grid_dependency_wait();
  xl_grid_launch_dependents();
  const int pos = *pos_ptr;
  if (pos < 0 || pos >= Smax) return;
  const int hd = H * D, half = D / 2;
  const long long total = (long long)B * H * half;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int d = 2 * (int)(i % half);
    const int h = (int)((i / half) % H);
    const int b = (int)(i / ((long long)half * H));
    T* q = qkv + (long long)b * ld + h * D + d;
    T* k = q + hd;
    const T* v = q + 2 * hd;
    float k0 = xl_to_float(k[0]), k1 = xl_to_float(k[1]);
    if (d < R) {
      const float sn = xl_to_float(sin_t[(long long)pos * (R / 2) + d / 2]);
      const float cs = xl_to_float(cos_t[(long long)pos * (R / 2) + d / 2]);
      const float q0 = xl_to_float(q[0]), q1 = xl_to_float(q[1]);
      q[0] = xl_from_float<T>(q0 * cs - q1 * sn);
      q[1] = xl_from_float<T>(q1 * cs + q0 * sn);
      const float r0 = k0 * cs - k1 * sn, r1 = k1 * cs + k0 * sn;
      k0 = r0;
      k1 = r1;
      k[0] = xl_from_float<T>(k0);
      k[1] = xl_from_float<T>(k1);
    }
    const long long dst = (((long long)b * H + h) * Smax + pos) * D + d;
    k_cache[dst] = xl_from_float<T>(k0);
    k_cache[dst + 1] = xl_from_float<T>(k1);
    v_cache[dst] = v[0];
    v_cache[dst + 1] = v[1];
  }
}

XL_API int xl_rotary_append(void* qkv, long long ld, const void* sin_t, const void* cos_t, void* k_cache, void* v_cache,
                            const int* pos_ptr, int B, int H, int D, int R, int Smax, int dtype, cudaStream_t s) {
  if ((D & 1) || (R & 1) || R > D) return -1;
  const long long total = (long long)B * H * (D / 2);
  const int grid = xl_grid_for(total, 256);
  XL_DISPATCH_DTYPE(dtype, T, {
    const cudaError_t e = xl_launch_overlapped(rotary_append_kernel<T>, dim3(grid), dim3(256), (size_t)0, s, (T*)qkv, ld, (const T*)sin_t,
                                               (const T*)cos_t, (T*)k_cache, (T*)v_cache, pos_ptr, B, H, D, R, Smax);
    if (e != cudaSuccess) return (int)e;
  });
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------------------------
// Keys and values of whole prompts into the caches: rows (b, s) of qkv hold [q | k | v], each heads x D; caches (B, H, Smax, D). Bound by
// HBM: 16-byte pieces, read in the order of the rows. (Two strided copies of 8192 x 4096 took 79 us each, both 40 us this way.)
// ------------------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    kv_fill_kernel(const uint4* __restrict__ qkv, uint32_t ld, uint4* __restrict__ k_cache, uint4* __restrict__ v_cache, uint32_t total,
                   uint32_t S, uint32_t H, uint32_t D, uint32_t Smax) {  // ld, D: in 16-byte pieces
  const uint32_t hd = H * D;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const uint32_t row = i / (2 * hd), c = i - row * 2 * hd;  // c: piece of [k | v]
    const uint32_t b = row / S, pos = row - b * S, f = c < hd ? c : c - hd, h = f / D;
    const uint4 v = qkv[(long long)row * ld + hd + c];
    (c < hd ? k_cache : v_cache)[(((long long)b * H + h) * Smax + pos) * D + (f - h * D)] = v;
  }
}
XL_API int xl_kv_fill(const void* qkv, long long ld, void* k_cache, void* v_cache, int B, int S, int H, int D, int Smax, int dtype,
                      cudaStream_t s) {
  const int n = dtype == XL_F32 ? 4 : 8;  // values per piece
  const long long total = (long long)B * S * 2 * H * D / n;
  if (B < 1 || S < 1 || S > Smax || H < 1 || D < n || D % n || ld % n || total > 0x7fffffffLL || ld / n > 0x7fffffffLL) return -1;
  if ((((uintptr_t)qkv) | ((uintptr_t)k_cache) | ((uintptr_t)v_cache)) & 15) return -1;
  kv_fill_kernel<<<xl_grid_for(total, 256 * 4), 256, 0, s>>>((const uint4*)qkv, (uint32_t)(ld / n), (uint4*)k_cache, (uint4*)v_cache,
                                                            (uint32_t)total, (uint32_t)S, (uint32_t)H, (uint32_t)(D / n), (uint32_t)Smax);
  return (int)cudaGetLastError();
}

// N consecutive elements (N * sizeof(T) a multiple of 16, p 16-byte aligned) through 128-bit accesses
template <typename T, int N> __device__ __forceinline__ void xl_load_vec(const T* __restrict__ p, float (&out)[N]) {
  constexpr int PER = 16 / sizeof(T);
#pragma unroll
  for (int q = 0; q < N / PER; ++q) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p + q * PER);
    const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
    for (int i = 0; i < PER; ++i) out[q * PER + i] = xl_to_float(e[i]);
  }
}
template <typename T, int N> __device__ __forceinline__ void xl_store_vec(T* __restrict__ p, const float (&in)[N]) {
  constexpr int PER = 16 / sizeof(T);
#pragma unroll
  for (int q = 0; q < N / PER; ++q) {
    uint4 raw;
    T* e = reinterpret_cast<T*>(&raw);
#pragma unroll
    for (int i = 0; i < PER; ++i) e[i] = xl_from_float<T>(in[q * PER + i]);
    *reinterpret_cast<uint4*>(p + q * PER) = raw;
  }
}

// ------------------------------------------------------------------------------------------------------------------
// Residual update + LayerNorm for a few rows: x += delta (+ bias); h = LayerNorm(x) * w + b. One CTA per row. What bounds it is one
// round trip to memory and the two sums over the CTA, so everything that is read is asked for at once and a sum takes one
// barrier (each warp adds the warps' sums up itself). 16 rows of 4096, delta and bias, in a chain of launches: 3.5 -> 2.4 us (weights read behind the
// statistics, sums by one thread between two barriers before).
// ------------------------------------------------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ void aln_unpack(const uint4& raw, float (&out)[8]) {
  const T* e = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int i = 0; i < 8; ++i) out[i] = xl_to_float(e[i]);
}
template <> __device__ __forceinline__ void aln_unpack<float>(const uint4&, float (&)[8]) {}

template <typename T, int VECS>  // VECS vectors of 8 elements per thread: cols <= 256 * 8 * VECS
__global__ void __launch_bounds__(256)
    add_layer_norm_kernel(T* x, const int* idx, const T* table, int table_rows, const T* delta, const T* bias, const T* w, const T* b, T* h,
                          int cols, float eps) {
  xl_grid_dependency_wait();
  xl_grid_launch_dependents();
  constexpr bool WIDE = sizeof(T) == 4;  // fp32 rows: two 16-byte pieces a vector, weights read where they are used
  __shared__ float red[2][8];
  const int row = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  T* xr = x + (long long)row * cols;
  const T* src = xr;
  if (idx) {  // the row comes from the table (zeros for an index outside it) and is stored
    const int r = idx[row];
    src = r >= 0 && r < table_rows ? table + (long long)r * cols : nullptr;
  }
  float v[VECS][8];
  uint4 raw[4][VECS];  // delta, bias, w, b
  const T* from[4] = {delta ? delta + (long long)row * cols : nullptr, bias, w, b};
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    const int c = (threadIdx.x + i * 256) * 8;
    if (c < cols) {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[i][e] = 0.f;
      if (src) xl_load_vec<T, 8>(src + c, v[i]);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (!WIDE && from[q]) raw[q][i] = *reinterpret_cast<const uint4*>(from[q] + c);
    }
  }
  auto operand = [&](int q, int i, int c, float (&out)[8]) {
    if constexpr (WIDE) xl_load_vec<T, 8>(from[q] + c, out);
    else aln_unpack<T>(raw[q][i], out);
  };
  auto block_sum = [&](float t, int k) {
    t = xl_warp_sum(t);
    if (lane == 0) red[k][warp] = t;
    __syncthreads();
    t = red[k][lane & 7];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
  };
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    const int c = (threadIdx.x + i * 256) * 8;
    if (c < cols) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (from[q]) {
          float d[8];
          operand(q, i, c, d);
#pragma unroll
          for (int e = 0; e < 8; ++e) v[i][e] += d[e];
        }
      }
      if (delta || bias || idx) {
        xl_store_vec<T, 8>(xr + c, v[i]);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[i][e] = xl_to_float(xl_from_float<T>(v[i][e]));  // what later readers of x see
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) sum += v[i][e];
    }
  }
  const float mean = block_sum(sum, 0) / cols;
  float sq = 0.f;
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    if ((threadIdx.x + i * 256) * 8 < cols) {
#pragma unroll
      for (int e = 0; e < 8; ++e) sq += (v[i][e] - mean) * (v[i][e] - mean);
    }
  }
  const float rstd = rsqrtf(block_sum(sq, 1) / cols + eps);
#pragma unroll
  for (int i = 0; i < VECS; ++i) {
    const int c = (threadIdx.x + i * 256) * 8;
    if (c < cols) {
      float wv[8], bv[8], o[8];
      operand(2, i, c, wv);
      operand(3, i, c, bv);
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = (v[i][e] - mean) * rstd * wv[e] + bv[e];
      xl_store_vec<T, 8>(h + (long long)row * cols + c, o);
    }
  }
}

static int aln_launch(void* x, const int* idx, const void* table, int table_rows, const void* delta, const void* bias, const void* w,
                      const void* b, void* h, int rows, int cols, float eps, int dtype, cudaStream_t s) {
  if (cols > 256 * 32 || (cols % 8) || rows < 1 || w == nullptr || b == nullptr) return -1;
  XL_DISPATCH_DTYPE(dtype, T, {
    void (*kernel)(T*, const int*, const T*, int, const T*, const T*, const T*, const T*, T*, int, float) =
        cols <= 256 * 8 ? add_layer_norm_kernel<T, 1> : (cols <= 256 * 16 ? add_layer_norm_kernel<T, 2> : add_layer_norm_kernel<T, 4>);
    const cudaError_t e = xl_launch_overlapped(kernel, dim3(rows), dim3(256), (size_t)0, s, (T*)x, idx, (const T*)table, table_rows,
                                               (const T*)delta, (const T*)bias, (const T*)w, (const T*)b, (T*)h, cols, eps);
    if (e != cudaSuccess) return (int)e;
  });
  return (int)cudaGetLastError();
}
// x (rows, cols) is updated in place when delta or bias is given; h (rows, cols) receives the normalised rows.
XL_API int xl_add_layer_norm(void* x, const void* delta, const void* bias, const void* w, const void* b, void* h,
                             int rows, int cols, float eps, int dtype, cudaStream_t s) {
  return aln_launch(x, nullptr, nullptr, 0, delta, bias, w, b, h, rows, cols, eps, dtype, s);
}
// x (rows, cols) = table[idx] (zeros for an index outside its table_rows), h the normalised rows; 16-byte aligned tables.
XL_API int xl_gather_layer_norm(const int* idx, const void* table, int table_rows, void* x, const void* w, const void* b, void* h,
                                int rows, int cols, float eps, int dtype, cudaStream_t s) {
  if (!idx || !table || (((uintptr_t)table) & 15)) return -1;
  return aln_launch(x, idx, table, table_rows, nullptr, nullptr, w, b, h, rows, cols, eps, dtype, s);
}

// ------------------------------------------------------------------------------------------------------------------
// Greedy sampling support: per row of logits (rows, V) the maximum and its index (+ index_offset of this vocabulary
// shard); pos_ptr, if given, is incremented by one afterwards (advances the decoding position on the device).
// ------------------------------------------------------------------------------------------------------------------
// One row per cluster of 1 to 8 CTAs: 16-byte loads (single elements up to the first and after the last 16-byte boundary of the
// row), the CTAs' winners meet in the shared memory of the first one. What bounds it is latency: one CTA per row kept 16 rows of
// 50400 16-bit logits on 16 SMs for 47 us (32000 fp32: 33 us); with eight CTAs per row a thread has three to four loads, all in
// flight together: 4.0 us (3.2 us). Of equal maxima the lowest index wins; NaN never wins.
// With `current` the choice is taken in the same launch: it becomes the row's current token and goes to row *pos + ahead - base of `buf`
// (where there is such a row), and with `advance` the CTA of the last row to finish moves the position on.
struct GreedyTake {
  int *current, *buf, *pos;
  int buf_rows, base, ahead, advance, rows;
  unsigned int* counter;  // zero between launches
};
struct ArgBest { float v; int i; };
__device__ __forceinline__ void arg_take(ArgBest& b, float v, int i) {
  if (v > b.v || (v == b.v && i < b.i)) { b.v = v; b.i = i; }
}
template <typename T>
__global__ void __launch_bounds__(256)
    argmax_rows_kernel(const T* logits, float* max_out, int* idx_out, int V, int valid, int index_offset, const GreedyTake take) {
  constexpr int N = XlVec<T>::N;
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int parts = (int)cluster.num_blocks(), part = (int)cluster.block_rank();
  __shared__ ArgBest warps[8], ctas[8];
  xl_grid_dependency_wait();
  const long long row = blockIdx.y;
  const T* p = logits + row * V;
  const int head = min(valid, (int)(((16 - ((uintptr_t)p & 15)) & 15) / sizeof(T)));
  const int vecs = (valid - head) / N, tail = head + vecs * N;
  ArgBest best{-INFINITY, 0};
  if (part == 0 && (int)threadIdx.x < head) arg_take(best, xl_to_float(p[threadIdx.x]), threadIdx.x);
#pragma unroll 4
  for (int i = part * 256 + threadIdx.x; i < vecs; i += parts * 256) {
    float v[N];
    xl_load16(p + head + i * N, v);
#pragma unroll
    for (int k = 0; k < N; ++k) arg_take(best, v[k], head + i * N + k);
  }
  if (part == 0 && tail + (int)threadIdx.x < valid) arg_take(best, xl_to_float(p[tail + threadIdx.x]), tail + threadIdx.x);
  auto warp_best = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float v = __shfl_xor_sync(0xffffffffu, best.v, o);
      const int i = __shfl_xor_sync(0xffffffffu, best.i, o);
      arg_take(best, v, i);
    }
  };
  warp_best();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) warps[warp] = best;
  __syncthreads();
  if (parts > 1) cluster.sync();  // every CTA of the cluster runs before its shared memory is written from outside
  if (warp == 0) {
    best = lane < 8 ? warps[lane] : ArgBest{-INFINITY, 0x7fffffff};
    warp_best();
    if (lane == 0) *(parts > 1 ? cluster.map_shared_rank(&ctas[part], 0) : &ctas[0]) = best;
  }
  if (parts > 1) cluster.sync();
  if (part == 0 && threadIdx.x == 0) {
    best = ctas[0];
    for (int k = 1; k < parts; ++k) arg_take(best, ctas[k].v, ctas[k].i);
    if (take.current) {
      const int at = *take.pos, r = at + take.ahead - take.base;
      take.current[row] = best.i;
      if (r >= 0 && r < take.buf_rows) take.buf[(long long)r * take.rows + row] = best.i;
      if (take.advance) {
        __threadfence();  // every row has read the position before the last one moves it
        if (atomicAdd(take.counter, 1u) == (unsigned int)take.rows - 1) {
          *take.counter = 0;
          *take.pos = at + 1;
        }
      }
    } else {
      max_out[row] = best.v;
      idx_out[row] = best.i + index_offset;
    }
  }
}
__global__ void advance_position_kernel(int* pos) {
  xl_grid_dependency_wait();
  xl_grid_launch_dependents();
  *pos += 1;
}

static int argmax_launch(const void* logits, float* max_out, int* idx_out, long long rows, int V, int valid, int index_offset,
                         const GreedyTake& take, int dtype, cudaStream_t s) {
  // two loads per thread and CTA are enough work; no more CTAs than four per SM together
  const int per_pass = 256 * (dtype == XL_F32 ? 4 : 8);
  int parts = 1;
  while (parts < 8 && valid > 2 * per_pass * parts && rows * parts * 2 <= 4 * 148) parts *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)parts, 1, 1);
  cfg.blockDim = dim3(256, 1, 1);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)parts;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  for (long long r0 = 0; r0 < rows; r0 += 65535) {  // rows are the y axis of the grid
    cfg.gridDim.y = (unsigned)(rows - r0 < 65535 ? rows - r0 : 65535);
    XL_DISPATCH_DTYPE(dtype, T, {
      const cudaError_t e = cudaLaunchKernelEx(&cfg, argmax_rows_kernel<T>, (const T*)logits + r0 * V, max_out ? max_out + r0 : nullptr,
                                               idx_out ? idx_out + r0 : nullptr, V, valid, index_offset, take);
      if (e != cudaSuccess) return (int)e;
    });
  }
  return (int)cudaGetLastError();
}
XL_API int xl_argmax_rows(const void* logits, float* max_out, int* idx_out, long long rows, int V, int valid,
                          int index_offset, int dtype, cudaStream_t s) {
  if (rows < 1) return 0;
  return argmax_launch(logits, max_out, idx_out, rows, V, valid, index_offset, GreedyTake{}, dtype, s);
}
// The greedy choice of every row taken (see GreedyTake): current (rows), buf (buf_rows, rows) int32, *pos the position. `counter`: a
// zero-initialised word (left zeroed). At most 65535 rows.
XL_API int xl_take_greedy(const void* logits, int* current, int* buf, int* pos, unsigned int* counter, int rows, int V, int valid,
                          int buf_rows, int base, int ahead, int advance, int dtype, cudaStream_t s) {
  if (rows < 1 || rows > 65535 || valid < 1 || valid > V || !current || !buf || !pos || !counter) return -1;
  return argmax_launch(logits, nullptr, nullptr, rows, V, valid, 0, GreedyTake{current, buf, pos, buf_rows, base, ahead, advance, rows, counter},
                       dtype, s);
}
XL_API int xl_advance_position(int* pos, cudaStream_t s) {
  const cudaError_t e = xl_launch_overlapped(advance_position_kernel, dim3(1), dim3(1), (size_t)0, s, pos);
  if (e != cudaSuccess) return (int)e;
  return (int)cudaGetLastError();
}

// buf: (rows, B) int32; writes vals (B) into row (*pos_ptr - base).
__global__ void store_row_kernel(int* buf, const int* pos_ptr, int base, const int* vals,
                                 int B, int rows) {
  xl_grid_dependency_wait();
  xl_grid_launch_dependents();
  const int r = *pos_ptr - base;
  if (r < 0 || r >= rows) return;
  for (int i = threadIdx.x; i < B; i += blockDim.x) buf[(long long)r * B + i] = vals[i];
}
XL_API int xl_store_row(int* buf, const int* pos_ptr, int base, const int* vals, int B, int rows, cudaStream_t s) {
  const cudaError_t e = xl_launch_overlapped(store_row_kernel, dim3(1), dim3(128), (size_t)0, s, buf, pos_ptr, base, vals, B, rows);
  if (e != cudaSuccess) return (int)e;
  return (int)cudaGetLastError();
}
