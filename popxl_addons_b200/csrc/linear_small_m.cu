// Linear layers of the decoding path, bf16 weights, few rows: C[M, N] = a[M, K] * w[N, K]^T, the weights streamed once.
// What follows the product in a layer happens in the epilogue, on the fp32 sums (M <= 64; `store` up to 128 rows):
//   store      C as bf16 or fp32
//   residual   x += mult * C (+ table[token]) on the fp32 residual stream; for the next layer h = DyT(x), or the first half of
//              an RMS norm: h = x * w and the sums of squares of x over blocks of 64 columns
//   swiglu     weight rows [gate | up]: y = silu(gate) * up
//   split_glu  weight rows [plain | gate | up]: plain results stored, a clamped gated unit of the others beside them
//   min_gru    weight rows [z | u | g], one row per sequence: one step of the recurrence on the fp32 state
//
// store and split_glu may take rows of such a half-done norm: their results are multiplied by 1 / sqrt(mean(x^2) + eps), summed
// up from the blocks' sums of squares while the weights arrive.
//
// The product is bandwidth-bound. The weight rows are the M = 128 operand of `tcgen05.mma` and the tokens (padded to 16, 32, 64 or
// 128) its N, so that one thread keeps the tensor core ahead of HBM: four instructions per 16 KB of weights, about 65 clocks each,
// are twice the rate at which an SM's share of the bandwidth arrives. TMA loads 128 x 64 blocks of weights, and the tokens' 64
// columns beside them, into a ring of 90 to 100 KB per CTA, two CTAs per SM. The two are CTAs of one product (K is split until
// both slots have one), or of a product that fills less than half of the slots and of its successor, whose ring fills while the
// product drains (programmatic dependent launch: weights that the previous kernel does not write are requested ahead of its end).
//
// A tile of 128 weight rows belongs to a cluster of KS CTAs (1 to 8), each with an equal range of K blocks; KS is what the SMs have
// room for. The CTAs leave their sums in shared memory, meet, and each finishes its share of the tile's results from the partial sums
// of all of them, added in CTA order, so results do not depend on timing. (Equal ranges of tiles x K blocks, one per CTA, with
// partial sums through global memory and the last arrival finishing a tile, took 2 to 10 us per launch more.) An epilogue
// that combines several weight rows per output channel (swiglu, min_gru) takes them
// into one tile: a tile is PARTS groups of CH channels, group p starting at weight row p * N / PARTS.
//
// Chains of launches on one B200, us (`mma.sync` with weights in registers and split K through global memory before -> now): 1 token
// 4096 x 4096 12.4 -> 8.4, 22016 x 4096 with swiglu 39.0 -> 32.3; 16 tokens 4096 x 11008 26.9 -> 18.0, 32000 x 4096 58.0 -> 43.0
// (6.1 TB/s); 40 tokens (tiles of 256 rows of the pair GEMM before) 2048 x 7680 30.5 -> 11.1, 12288 x 4096 29.6 -> 21.1,
// 32000 x 4096 57.0 -> 47.2. Epilogues of 17 to 64 tokens against plain products and kernels of their own: 40 tokens, width 2048
// split_glu 17.0 -> 15.6, residual with RMS norm 11.8 -> 10.7, swiglu 14.7 -> 12.9, min_gru 14.6 -> 10.5; 64 tokens, width 4096
// 50.3 -> 46.6, 25.9 -> 22.3, 38.6 -> 36.6, 31.1 -> 25.8.
//
// Roles per CTA: warp 0 loads, warp 1 allocates TMEM and issues the MMAs, warps 2-5 (above 32 tokens 2-9) drain the accumulator. Every wait is bounded; a role
// that gives up records a code in `*err`, all threads meet at the cluster's barriers and TMEM is freed.
#include "common.cuh"
#include "tcgen05.cuh"

#include <math.h>

namespace {

using namespace xl_tc;

constexpr int SM_KC = 64;            // k values per block: one 128-byte swizzle row

enum SmMode : int { SM_STORE = 0, SM_RESIDUAL = 1, SM_SWIGLU = 2, SM_MINGRU = 3, SM_SPLIT_GLU = 4 };

// split_glu has two kinds of tiles: first those of the plain rows (one part of 128 channels), then those of the gated unit.
template <int MODE> struct SmTile {
  static constexpr int PARTS = MODE == SM_SWIGLU || MODE == SM_SPLIT_GLU ? 2 : (MODE == SM_MINGRU ? 3 : 1);
  static constexpr int CH = PARTS == 2 ? 64 : (MODE == SM_MINGRU ? 40 : 128);  // channels per tile
  static constexpr int COLS = PARTS * CH;  // rows of the MMA that hold weights (120 of 128 for min_gru)
};
// NTOK: columns of the MMA, the tokens padded
template <int NTOK> struct SmRing {
  static constexpr int W_BYTES = 128 * SM_KC * 2, A_BYTES = NTOK * SM_KC * 2, STAGE = W_BYTES + A_BYTES;
  static constexpr int STAGES = NTOK <= 32 ? 5 : (NTOK == 64 ? 4 : 3);
  static constexpr int SMEM = STAGES * STAGE + 1024 /*alignment slack*/;
  // threads of the epilogue: one per TMEM lane, or two where many results are to be finished (40 tokens, 4096 x 12288 min_gru 24.7 -> 23.1
  // us, 16384 x 2048 split_glu 16.2 -> 15.6; 24 tokens, 3072 x 1024 min_gru 7.1 -> 8.5)
  static constexpr int EPI = NTOK > 32 ? 256 : 128;
  static constexpr uint32_t TMEM_COLS = NTOK < 32 ? 32 : NTOK;
  static_assert(NTOK * 132 * 4 <= STAGES * STAGE, "the partial sums take the ring's place");
};
enum { ERR_SM_FULL = 31, ERR_SM_EMPTY = 32, ERR_SM_ACC_FULL = 33 };

struct SmParams {
  const __nv_bfloat16* a;
  long long lda;
  const __nv_bfloat16* w;  // (N, K), contiguous
  int M, N, K;
  // store / swiglu / min_gru
  void* y;
  long long ldy;
  int y_f32;
  // residual
  float* x;
  float mult;
  const int* tokens;
  const __nv_bfloat16* table;
  int vocab;
  const float *alpha, *nw, *nb;  // DyT; alpha null: h = x * nw and the sums of squares
  __nv_bfloat16* h;
  float* sumsq_out;  // (M, column tiles)
  // store / split_glu: sums of squares of the rows of a half-done norm, (M, sumsq_parts), or null
  const float* sumsq;
  int sumsq_parts;
  float eps;
  // split_glu: y holds the plain results, z the unit's
  int cols;
  __nv_bfloat16* z;
  long long ldz;
  float limit, slope, shift;
  // min_gru
  const float *bz, *bu;
  float* state;
  const int *pos, *count;
  int ksplit;  // CTAs of a cluster
  int read_ahead;  // the weights were complete before the previous launch
  int* err;
};

__device__ __forceinline__ float sigmoid_f(float v) { return 1.f / (1.f + expf(-v)); }
__device__ __forceinline__ float silu_f(float v) { return v / (1.f + expf(-v)); }

// Four channels c .. c + 3 of row r (those below `channels`). All loads come before the first store: their latencies overlap.
// Returns the sum of squares of what it wrote to the residual stream.
template <int MODE>
__device__ __forceinline__ float sm_epilogue(const SmParams& p, int r, int c, const float (&v)[SmTile<MODE>::PARTS][4], int channels,
                                             bool unit) {
  constexpr int LAST = SmTile<MODE>::PARTS - 1;
  const int n = min(4, channels - c);
  float sq = 0.f;
  const long long at = (long long)r * channels + c, yat = (long long)r * p.ldy + c;
  if (MODE == SM_SPLIT_GLU && unit) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (e < n)
        p.z[(long long)r * p.ldz + c + e] =
            __float2bfloat16_rn(xl_clamped_glu_value(v[0][e], v[LAST][e], p.limit, p.slope, p.shift));
  } else if (MODE == SM_STORE || MODE == SM_SPLIT_GLU) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (e < n) {
        if (p.y_f32) ((float*)p.y)[yat + e] = v[0][e];
        else ((__nv_bfloat16*)p.y)[yat + e] = __float2bfloat16_rn(v[0][e]);
      }
    }
  } else if (MODE == SM_RESIDUAL) {
    float x[4], add[4], nw[4], nb[4];
    const __nv_bfloat16* row = p.table ? p.table + (long long)min(max(p.tokens[r], 0), p.vocab - 1) * channels + c : nullptr;
    const float alpha = p.alpha ? *p.alpha : 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = e < n ? e : 0;
      x[e] = p.x[at + k];
      add[e] = row ? __bfloat162float(row[k]) : 0.f;
      nw[e] = p.nw ? p.nw[c + k] : 0.f;
      nb[e] = p.alpha ? p.nb[c + k] : 0.f;
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (e < n) {
        const float s = x[e] + p.mult * v[0][e] + add[e];
        p.x[at + e] = s;
        sq += s * s;
        if (p.alpha) p.h[at + e] = __float2bfloat16_rn(tanhf(alpha * s) * nw[e] + nb[e]);
        else if (p.nw) p.h[at + e] = __float2bfloat16_rn(s * nw[e]);
      }
    }
  } else if (MODE == SM_SWIGLU) {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      if (e < n) ((__nv_bfloat16*)p.y)[yat + e] = __float2bfloat16_rn(silu_f(v[0][e]) * v[LAST][e]);
  } else {
    float old[4], bz[4], bu[4];
    const bool fresh = p.pos[r] <= 0, real = p.count[r] > 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = e < n ? e : 0;
      old[e] = fresh ? 0.f : p.state[at + k];
      bz[e] = p.bz[c + k];
      bu[e] = p.bu[c + k];
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (e < n) {
        const float z = sigmoid_f(v[0][e] + bz[e]), u = v[1 % SmTile<MODE>::PARTS][e] + bu[e];
        float s = old[e];
        if (real) {
          s = (1.f - z) * s + z * (u >= 0.f ? u + 0.5f : sigmoid_f(u));
          p.state[at + e] = s;
        }
        ((__nv_bfloat16*)p.y)[yat + e] = __float2bfloat16_rn(s * silu_f(v[LAST][e]));
      }
    }
  }
  return sq;
}

__device__ __forceinline__ float4 ld_cluster_v4(uint32_t cluster_addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(cluster_addr));
  return v;
}

template <int MODE, int NTOK>
__global__ void __launch_bounds__(64 + SmRing<NTOK>::EPI, 2)
    linear_small_m_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, const SmParams p) {
  using L = SmTile<MODE>;
  using R = SmRing<NTOK>;
  constexpr int COLS = L::COLS, CH = L::CH, PARTS = L::PARTS, STAGES = R::STAGES, SM_EPI = R::EPI;
  constexpr int RED_LD = 132;
  extern __shared__ uint8_t smem_raw[];
  __shared__ float row_scale[NTOK];
  __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  uint8_t* ring = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);  // the same offset in every CTA of the cluster
  volatile int* abort_flag = &abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunks = (p.K + SM_KC - 1) / SM_KC;
  // tiles [0, plain) have one part of 128 channels (split_glu only), the others PARTS parts of CH
  const int plain = MODE == SM_SPLIT_GLU ? (p.cols + 127) / 128 : 0;
  const int channels = MODE == SM_SPLIT_GLU ? (p.N - p.cols) / PARTS : p.N / PARTS;
  const int tile = blockIdx.x / p.ksplit, rank = blockIdx.x - tile * p.ksplit;  // clusters are consecutive CTAs
  const int kb0 = chunks * rank / p.ksplit, blocks = chunks * (rank + 1) / p.ksplit - kb0;  // at least one

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_full, 1);
    abort_word = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    tmem_alloc(&tmem_slot, R::TMEM_COLS);
    tmem_relinquish();
  }
  tcgen05_fence_before();
  __syncthreads();
  tcgen05_fence_after();
  const uint32_t tmem_base = tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------ loads --------------------------------------------------------
    if (elect_one()) {
      const bool one = MODE == SM_SPLIT_GLU && tile < plain;
      const int n0 = MODE == SM_SPLIT_GLU ? (one ? tile * 128 : p.cols + (tile - plain) * CH) : tile * CH;
      auto load_w = [&](int i, int s) {
#pragma unroll
        for (int q = 0; q < PARTS; ++q)  // boxes of CH rows; a plain tile's are consecutive
          tma_load_2d(ring + s * R::STAGE + q * CH * 128, &map_w, &full_bar[s], (kb0 + i) * SM_KC, n0 + q * (one ? CH : channels));
      };
      auto load_a = [&](int i, int s) { tma_load_2d(ring + s * R::STAGE + R::W_BYTES, &map_a, &full_bar[s], (kb0 + i) * SM_KC, 0); };
      constexpr uint32_t BYTES = COLS * 128 + R::A_BYTES;
      const int ahead = min(STAGES, blocks);
      if (!p.read_ahead) xl_grid_dependency_wait();
      for (int i = 0; i < ahead; ++i) {
        mbar_expect_tx(&full_bar[i], BYTES);
        load_w(i, i);
      }
      xl_grid_dependency_wait();  // the first weights are on their way; everything else may come from the previous kernel
      xl_grid_launch_dependents();
      for (int i = 0; i < ahead; ++i) load_a(i, i);
      uint32_t stage = 0, phase = 0;
      for (int i = ahead; i < blocks; ++i) {
        if (!mbar_wait(&empty_bar[stage], phase, abort_flag, p.err, ERR_SM_EMPTY)) break;
        mbar_expect_tx(&full_bar[stage], BYTES);
        load_w(i, stage);
        load_a(i, stage);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------ MMAs ---------------------------------------------------------
    xl_grid_dependency_wait();  // the tokens arrive after it: no bounded wait runs while the predecessor still does
    if (elect_one()) {
      constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(NTOK >> 3) << 17) | (8u << 24);
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      for (int i = 0; i < blocks; ++i) {
        ok = mbar_wait(&full_bar[stage], phase, abort_flag, p.err, ERR_SM_FULL);
        if (!ok) break;
        tcgen05_fence_after();
        const uint32_t sw = smem_u32(ring + stage * R::STAGE), sa = sw + R::W_BYTES;
#pragma unroll
        for (int k = 0; k < SM_KC / 16; ++k)
          tcgen05_mma_f16(tmem_base, make_smem_desc(sw + k * 32, 16), make_smem_desc(sa + k * 32, 16), idesc, (i | k) != 0 ? 1u : 0u);
        tcgen05_commit(&empty_bar[stage]);
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (ok) tcgen05_commit(&acc_full);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------ partial sums -> shared memory --------------------------------
    xl_grid_dependency_wait();
    xl_grid_launch_dependents();
    const int q4 = warp & 3, row = q4 * 32 + lane;  // TMEM lane = weight row of the tile
    float* red = reinterpret_cast<float*>(ring);    // [token][weight row]: every load of the ring has been read by an MMA by then
    if ((MODE == SM_STORE || MODE == SM_SPLIT_GLU) && p.sumsq) {  // while the weights arrive
      const int et = threadIdx.x - 64;
      for (int r0 = 0; r0 < p.M; r0 += SM_EPI / 8) {  // eight lanes add a row's parts up
        const int r = r0 + (et >> 3);
        float sq = 0.f;
        if (r < p.M) {
#pragma unroll 8
          for (int i = et & 7; i < p.sumsq_parts; i += 8) sq += p.sumsq[(long long)r * p.sumsq_parts + i];
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if ((et & 7) == 0 && r < p.M) row_scale[r] = 1.f / sqrtf(sq / p.K + p.eps);
      }
    }
    if (mbar_wait_warp(&acc_full, 0, abort_flag, p.err, ERR_SM_ACC_FULL)) {
      tcgen05_fence_after();
#pragma unroll 1
      for (int t0 = (warp - 2) / 4 * 16; t0 < NTOK && t0 < p.M; t0 += SM_EPI / 8) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(tmem_base + ((uint32_t)(q4 * 32) << 16) + t0, r);
        tmem_ld_wait();
#pragma unroll
        for (int t = 0; t < 16; ++t) red[(t0 + t) * RED_LD + row] = __uint_as_float(r[t]);
      }
    }
    tcgen05_fence_before();
  }
  __syncthreads();
  if (p.ksplit > 1) {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  if (warp >= 2 && !*abort_flag) {
    // ------------------------------------------------ results ------------------------------------------------------
    const int et = threadIdx.x - 64;
    const bool unit = tile >= plain;  // one part of 128 channels, or PARTS parts of CH
    const int ch = MODE == SM_SPLIT_GLU && !unit ? 128 : CH, parts = MODE == SM_SPLIT_GLU && !unit ? 1 : PARTS;
    const int end = MODE == SM_SPLIT_GLU && !unit ? p.cols : channels, per_row = ch / 4;
    uint32_t red_at[8];  // this CTA's and its peers' partial sums
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (k < p.ksplit) asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(red_at[k]) : "r"(smem_u32(ring)), "r"(k));
    for (int i = rank * SM_EPI + et; i < p.M * per_row; i += p.ksplit * SM_EPI) {
      const int r = i / per_row, cc = (i - r * per_row) * 4, c = (unit ? tile - plain : tile) * ch + cc;
      float sq = 0.f;
      if (c < end) {
        float v[PARTS][4];
#pragma unroll
        for (int q = 0; q < PARTS; ++q) {
          float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
          if (MODE != SM_SPLIT_GLU || q < parts) {
            const uint32_t off = (uint32_t)(r * RED_LD + q * CH + cc) * 4;
            float4 part[8];
#pragma unroll
            for (int k = 0; k < 8; ++k)
              if (k < p.ksplit) part[k] = ld_cluster_v4(red_at[k] + off);
            t = part[0];
#pragma unroll
            for (int k = 1; k < 8; ++k)
              if (k < p.ksplit) { t.x += part[k].x; t.y += part[k].y; t.z += part[k].z; t.w += part[k].w; }
          }
          v[q][0] = t.x; v[q][1] = t.y; v[q][2] = t.z; v[q][3] = t.w;
          if ((MODE == SM_STORE || MODE == SM_SPLIT_GLU) && p.sumsq) {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[q][e] *= row_scale[r];
          }
        }
        sq = sm_epilogue<MODE>(p, r, c, v, end, unit);
      }
      if (MODE == SM_RESIDUAL && p.sumsq_out) {
        // a half-warp holds 64 columns of one row, the warp two such blocks; all lanes are here
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if ((lane & 15) == 0 && c < end) p.sumsq_out[(long long)r * ((p.N + 63) / 64) + c / 64] = sq;
      }
    }
  }
  __syncwarp();
  if (p.ksplit > 1) {  // the peers may still read this CTA's sums
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
  if (warp == 1) {
    tcgen05_fence_after();
    tmem_dealloc(tmem_base, R::TMEM_COLS);
  }
}

template <int MODE, int NTOK> int sm_launch_tokens(SmParams p, int sms, cudaStream_t s) {
  using L = SmTile<MODE>;
  using R = SmRing<NTOK>;
  const int paired = MODE == SM_SPLIT_GLU ? p.N - p.cols : p.N;
  if (paired % L::PARTS) return -1;
  const int plain = MODE == SM_SPLIT_GLU ? (p.cols + 127) / 128 : 0;
  const int channels = paired / L::PARTS, chunks = (p.K + SM_KC - 1) / SM_KC, n_tiles = plain + (channels + L::CH - 1) / L::CH;
  static XlPerDevice smem;
  XL_TRY(xl_allow_smem(linear_small_m_kernel<MODE, NTOK>, R::SMEM, smem));
  // A power of two that two CTAs per SM have room for, at most eight. Room for one CTA per SM only was slower (16 tokens, 4096 x
  // 11008: 20.6 us with 4 CTAs per cluster, 18.0 with 8; 12288 x 4096: 22.5 with 1, 19.6 with 2), and so were clusters of 6 and 3
  // (6144 x 4096: 15.9 us with 6, 11.9 with 4; 12288 x 4096: 25.3 with 3).
  p.ksplit = 1;
  while (p.ksplit < 8 && 2 * p.ksplit * n_tiles <= 2 * sms && 4 * p.ksplit <= chunks) p.ksplit *= 2;
  CUtensorMap mw, ma;
  int rc = make_map_bf16(&mw, p.w, p.N, p.K, p.K, L::CH);
  if (rc == 0) rc = make_map_bf16(&ma, p.a, p.M, p.K, p.lda, NTOK);
  if (rc) return rc == -2 ? (int)cudaErrorNotSupported : (int)cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(n_tiles * p.ksplit));
  cfg.blockDim = dim3(64 + R::EPI);
  cfg.dynamicSmemBytes = R::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)p.ksplit;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, linear_small_m_kernel<MODE, NTOK>, mw, ma, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}
template <int MODE> int sm_launch(const SmParams& p, int sms, cudaStream_t s) {
  if (p.M <= 16) return sm_launch_tokens<MODE, 16>(p, sms, s);
  if (p.M <= 32) return sm_launch_tokens<MODE, 32>(p, sms, s);
  if (MODE != SM_STORE || p.M <= 64) return sm_launch_tokens<MODE, 64>(p, sms, s);
  return sm_launch_tokens<SM_STORE, 128>(p, sms, s);
}

int sm_check(const void* a, long long lda, const void* w, int M, int N, int K, int max_m = 64) {
  if (M < 1 || M > max_m || N < 1 || K < 8 || (K % 8) || (lda % 8) || lda < K) return -1;
  if (((uintptr_t)a & 15) || ((uintptr_t)w & 15)) return -1;
  return 0;
}

}  // namespace

// All: a (M, K) bf16 with row stride lda (a multiple of 8), w (N, K) bf16 contiguous, M <= 64 (xl_linear_small_m: 128), K a multiple
// of 8; returns -1 for arguments the kernel does not take. read_ahead: w was complete before the previous launch on the stream. y
// (M, N) with row stride ldy, bf16 or fp32. sumsq (M, sumsq_parts), or null: the rows of y are multiplied by
// 1 / sqrt(sum of the row's sumsq / K + eps).
XL_API int xl_linear_small_m(const void* a, long long lda, const void* w, void* y, long long ldy, int y_f32, const float* sumsq,
                             int sumsq_parts, float eps, int M, int N, int K, int sms, int read_ahead, int* err,
                             cudaStream_t s) {
  if (sm_check(a, lda, w, M, N, K, 128) || !y || (sumsq && sumsq_parts < 1)) return -1;
  SmParams p = {};
  p.a = (const __nv_bfloat16*)a; p.lda = lda; p.w = (const __nv_bfloat16*)w; p.M = M; p.N = N; p.K = K;
  p.y = y; p.ldy = ldy; p.y_f32 = y_f32; p.sumsq = sumsq; p.sumsq_parts = sumsq_parts; p.eps = eps;
  p.read_ahead = read_ahead; p.err = err;
  return sm_launch<SM_STORE>(p, sms, s);
}

// w rows [cols plain | F gate | F up], N = cols + 2F: y (M, cols) with row stride ldy and z (M, F) with row stride ldz, bf16;
// sumsq as in xl_linear_small_m.
XL_API int xl_linear_small_m_split_glu(const void* a, long long lda, const void* w, void* y, long long ldy, int cols, void* z,
                                       long long ldz, float limit, float slope, float shift, const float* sumsq, int sumsq_parts,
                                       float eps, int M, int N, int K, int sms, int read_ahead, int* err,
                                       cudaStream_t s) {
  if (sm_check(a, lda, w, M, N, K) || cols < 0 || cols > N || (cols && !y) || (cols < N && !z) ||
      (sumsq && sumsq_parts < 1))
    return -1;
  SmParams p = {};
  p.a = (const __nv_bfloat16*)a; p.lda = lda; p.w = (const __nv_bfloat16*)w; p.M = M; p.N = N; p.K = K;
  p.y = y; p.ldy = ldy; p.cols = cols; p.z = (__nv_bfloat16*)z; p.ldz = ldz; p.limit = limit; p.slope = slope; p.shift = shift;
  p.sumsq = sumsq; p.sumsq_parts = sumsq_parts; p.eps = eps; p.read_ahead = read_ahead; p.err = err;
  return sm_launch<SM_SPLIT_GLU>(p, sms, s);
}

// x (M, N) fp32 += mult * a w^T; with nw, h (M, N) bf16 = x * nw and sumsq (M, ceil(N / 64)) = sums of x^2 over 64 columns.
XL_API int xl_linear_small_m_residual_rms(const void* a, long long lda, const void* w, float* x, float mult, const float* nw,
                                          void* h, float* sumsq, int M, int N, int K, int sms, int read_ahead, int* err,
                                          cudaStream_t s) {
  if (sm_check(a, lda, w, M, N, K) || !x || (nw && (!h || !sumsq))) return -1;
  SmParams p = {};
  p.a = (const __nv_bfloat16*)a; p.lda = lda; p.w = (const __nv_bfloat16*)w; p.M = M; p.N = N; p.K = K;
  p.x = x; p.mult = mult; p.nw = nw; p.h = (__nv_bfloat16*)h; p.sumsq_out = nw ? sumsq : nullptr;
  p.read_ahead = read_ahead; p.err = err;
  return sm_launch<SM_RESIDUAL>(p, sms, s);
}

// x (M, N) fp32 += mult * a w^T (+ table[tokens]); with alpha, h (M, N) bf16 = tanh(alpha x) nw + nb.
XL_API int xl_linear_small_m_residual(const void* a, long long lda, const void* w, float* x, float mult, const int* tokens,
                                      const void* table, int vocab, const float* alpha, const float* nw, const float* nb,
                                      void* h, int M, int N, int K, int sms, int read_ahead, int* err,
                                      cudaStream_t s) {
  if (sm_check(a, lda, w, M, N, K) || !x || (table && (!tokens || vocab < 1)) || (alpha && (!nw || !nb || !h)))
    return -1;
  SmParams p = {};
  p.a = (const __nv_bfloat16*)a; p.lda = lda; p.w = (const __nv_bfloat16*)w; p.M = M; p.N = N; p.K = K;
  p.x = x; p.mult = mult; p.tokens = tokens; p.table = (const __nv_bfloat16*)table; p.vocab = vocab;
  p.alpha = alpha; p.nw = nw; p.nb = nb; p.h = (__nv_bfloat16*)h; p.read_ahead = read_ahead; p.err = err;
  return sm_launch<SM_RESIDUAL>(p, sms, s);
}

// w rows [gate | up] (2F, K); y (M, F) bf16 contiguous.
XL_API int xl_linear_small_m_swiglu(const void* a, long long lda, const void* w, void* y, int M, int F, int K, int sms,
                                    int read_ahead, int* err, cudaStream_t s) {
  if (sm_check(a, lda, w, M, 2 * F, K) || !y) return -1;
  SmParams p = {};
  p.a = (const __nv_bfloat16*)a; p.lda = lda; p.w = (const __nv_bfloat16*)w; p.M = M; p.N = 2 * F; p.K = K;
  p.y = y; p.ldy = F; p.read_ahead = read_ahead; p.err = err;
  return sm_launch<SM_SWIGLU>(p, sms, s);
}

// w rows [z | u | g] (3W, K); row r is the next token of sequence r: state (M, W) fp32 advances where count[r] > 0 and starts
// from zero at pos[r] == 0; y (M, W) bf16 contiguous.
XL_API int xl_linear_small_m_min_gru(const void* a, long long lda, const void* w, const float* bz, const float* bu, float* state,
                                     const int* pos, const int* count, void* y, int M, int W, int K, int sms, int read_ahead, int* err,
                                     cudaStream_t s) {
  if (sm_check(a, lda, w, M, 3 * W, K) || !y || !state || !bz || !bu || !pos || !count) return -1;
  SmParams p = {};
  p.a = (const __nv_bfloat16*)a; p.lda = lda; p.w = (const __nv_bfloat16*)w; p.M = M; p.N = 3 * W; p.K = K;
  p.y = y; p.ldy = W; p.bz = bz; p.bu = bu; p.state = state; p.pos = pos; p.count = count; p.read_ahead = read_ahead; p.err = err;
  return sm_launch<SM_MINGRU>(p, sms, s);
}
