// Decode attention: one query per (b, h) against the cached keys and values of positions [0, pos], one launch; optionally with the
// rotation of the new query and key and the append of the new key and value in front of it.
//
// The positions of a (b, h) are consecutive memory, so a producer warp brings a stage of keys and as much of values at a time with two plain
// bulk copies into a ring of three stages. Cached positions do not depend on the previous kernel as a rule; they are then on their way
// before it ends. W = 8, 4 or 2 warps take a share of each stage (W = 8: 16 KB of keys, which is 32, 64 or 128 positions of 256, 128 or
// 64 features, and 96 KB of ring per CTA): a position is a group of 32, 16 or 8 lanes, 16 bytes of a key per lane, and every group has an
// online softmax of its own. The new key and value come from the projections: the CTA of the last positions rotates and appends them and
// takes them from registers.
// Grid (B * H, splits): CTAs that share a (b, h) leave (max, sum, unnormalised output) of their positions; the last one to finish
// (a counter per (b, h), left at zero again) merges them in order.
//
// What bounds it is HBM, and for short caches the latency of the chain load - score - softmax - merge, so splits are few (chosen by the
// caller), and where there are more CTAs than two per SM they are smaller, so that more chains run side by side (W by the caller, with
// the figures). Chains of launches on one B200, us (rotation and append as a kernel of their own, keys and values through registers -> here):
//   16 sequences of 528 positions, 16 heads of 256   37.3 -> 24.9 (5.6 TB/s)      1 sequence of 93, 16 heads of 128     7.3 -> 3.3
//   16 of 528, 16 heads of 128                       20.3 -> 14.6                 1 of 2000, 16 heads of 256           37.2 -> 9.5
//   16 of 1000, 32 heads of 64                       36.7 -> 26.6                 1 of 8000, 8 heads of 256            41.8 -> 15.5
//   300 of 100, 8 heads of 64                        23.9 -> 17.4                 128 of 60, 16 heads of 64            13.8 -> 9.7
#include "common.cuh"
#include "tcgen05.cuh"

#include <math.h>

namespace {

using namespace xl_tc;

constexpr int AD_UNROLL = 4;
enum { ERR_AD_FULL = 64, ERR_AD_EMPTY = 65 };

template <int D, int W> struct AdCfg {
  static constexpr int THREADS = (W + 1) * 32, CTAS = W == 8 ? 2 : 16 / W;  // per SM
  static constexpr int LANES = D / 8, GROUPS = 32 / LANES;  // lanes of a position, positions of a warp at a time
  static constexpr int POS = W * AD_UNROLL * GROUPS, ROW = D * 2, HALF = POS * ROW, STAGE = 2 * HALF, STAGES = 3;
  static constexpr int SMEM = STAGES * STAGE + 128 /*alignment slack*/;
};

struct AdParams {
  const void* qkv;  // rows of ldq: q (, k, v with `append`) of the new tokens, heads x D each
  long long ldq;
  void *k_cache, *v_cache;  // (B, H, Smax, D)
  void* out;
  long long ldo;
  float* part;
  unsigned int* counters;
  const int* pos;
  const void *sin_t, *cos_t;  // (Smax, R / 2)
  int H, Smax, R, append, read_ahead;
  float scale;
  int* err;
};

template <typename T> struct alignas(16) AdVec { T v[8]; };

__device__ __forceinline__ void ad_bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src),
               "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
template <int W> __device__ __forceinline__ void ad_sync() { asm volatile("bar.sync 1, %0;" ::"n"(W * 32) : "memory"); }

// W: warps that attend
template <typename T, int D, int W>
__global__ void __launch_bounds__((AdCfg<D, W>::THREADS), (AdCfg<D, W>::CTAS)) attn_decode_kernel(const __grid_constant__ AdParams p) {
  using C = AdCfg<D, W>;
  using Vec = AdVec<T>;
  constexpr int LANES = C::LANES, GROUPS = C::GROUPS, STREAMS = W * GROUPS;
  extern __shared__ uint8_t ad_smem[];
  __shared__ uint64_t full_bar[C::STAGES], empty_bar[C::STAGES];
  __shared__ int abort_word;
  __shared__ float sm[STREAMS], sl[STREAMS];
  __shared__ __align__(16) float so[STREAMS][D];
  __shared__ unsigned int is_last;
  uint8_t* ring = (uint8_t*)(((uintptr_t)ad_smem + 127) & ~(uintptr_t)127);
  volatile int* abort_flag = &abort_word;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = lane / LANES, at_d = lane % LANES * 8;
  const int bh = blockIdx.x, split = blockIdx.y, splits = gridDim.y, b = bh / p.H, h = bh % p.H;
  if (threadIdx.x == 0) {
    for (int s = 0; s < C::STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], W);
    }
    abort_word = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  T* const kb = (T*)p.k_cache + (long long)bh * p.Smax * D;
  T* const vb = (T*)p.v_cache + (long long)bh * p.Smax * D;
  // positions of this CTA: cached ones [first, cached_end), and the new one if `fresh`
  int pos, first, cached_end;
  bool fresh, rotate;
  auto range = [&]() {
    pos = *p.pos;
    const bool here = p.append && pos >= 0 && pos < p.Smax;
    const int cached = min(max(p.append ? pos : pos + 1, 0), p.Smax), len = cached + (here ? 1 : 0);
    const int per = (len + splits - 1) / splits;
    first = split * per;
    const int end = min(len, first + per);
    cached_end = min(cached, end);
    rotate = here && p.R > 0;
    fresh = here && first < end && end == len;
  };

  if (warp == W) {
    if (elect_one()) {
      if (!p.read_ahead) xl_grid_dependency_wait();
      range();
      auto load = [&](int at, int s) {
        const uint32_t bytes = (uint32_t)min(C::POS, cached_end - at) * C::ROW;
        mbar_expect_tx(&full_bar[s], 2 * bytes);
        ad_bulk_load(ring + s * C::STAGE, kb + (long long)at * D, bytes, &full_bar[s]);
        ad_bulk_load(ring + s * C::STAGE + C::HALF, vb + (long long)at * D, bytes, &full_bar[s]);
      };
      int at = first;
      for (int s = 0; s < C::STAGES && at < cached_end; ++s, at += C::POS) load(at, s);
      xl_grid_dependency_wait();  // no bounded wait runs while the previous kernel still does
      int stage = 0;
      uint32_t phase = 0;
      for (; at < cached_end; at += C::POS) {
        if (!mbar_wait(&empty_bar[stage], phase, abort_flag, p.err, ERR_AD_EMPTY)) break;
        load(at, stage);
        if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
      }
      if (*abort_flag)
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);  // copies in flight arrive before the CTA gives its memory back
    }
    return;
  }
  xl_grid_dependency_wait();
  xl_grid_launch_dependents();
  range();
  const T* row = (const T*)p.qkv + (long long)b * p.ldq + h * D + at_d;
  const bool newest = fresh && warp == W - 1;  // its first group takes the new position
  Vec qv = *reinterpret_cast<const Vec*>(row), kn, vn;
  if (newest) {
    kn = *reinterpret_cast<const Vec*>(row + p.H * D);
    vn = *reinterpret_cast<const Vec*>(row + 2 * p.H * D);
  }
  if (rotate) {
    const long long at = (long long)pos * (p.R / 2) + at_d / 2;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (at_d + 2 * e < p.R) {
        const float sn = xl_to_float(((const T*)p.sin_t)[at + e]), cs = xl_to_float(((const T*)p.cos_t)[at + e]);
        auto turn = [&](Vec& x) {
          const float x0 = xl_to_float(x.v[2 * e]), x1 = xl_to_float(x.v[2 * e + 1]);
          x.v[2 * e] = xl_from_float<T>(x0 * cs - x1 * sn);
          x.v[2 * e + 1] = xl_from_float<T>(x1 * cs + x0 * sn);
        };
        turn(qv);
        if (newest) turn(kn);
      }
    }
  }
  float q[8], o[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    q[e] = xl_to_float(qv.v[e]) * p.scale;
    o[e] = 0.f;
  }
  float m = -INFINITY, l = 0.f;
  if (newest) {
    float d = 0.f;
#pragma unroll
    for (int e = 0; e < 8; ++e) d += q[e] * xl_to_float(kn.v[e]);
#pragma unroll
    for (int off = LANES / 2; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
    if (group == 0) {
      const long long at = (long long)pos * D + at_d;
      *reinterpret_cast<Vec*>(kb + at) = kn;
      *reinterpret_cast<Vec*>(vb + at) = vn;
      m = d;
      l = 1.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] = xl_to_float(vn.v[e]);
    }
  }
  int stage = 0;
  uint32_t phase = 0;
  for (int at = first; at < cached_end; at += C::POS) {
    if (!__all_sync(0xffffffffu, mbar_wait(&full_bar[stage], phase, abort_flag, p.err, ERR_AD_FULL))) break;
    const int count = min(C::POS, cached_end - at), w0 = warp * AD_UNROLL * GROUPS, s0 = w0 + group;  // unit u: s0 + u * GROUPS
    if (w0 < count) {
      const uint8_t* st = ring + stage * C::STAGE + at_d * 2;
      Vec kk[AD_UNROLL], vv[AD_UNROLL];  // duplicates of the last position are masked below
#pragma unroll
      for (int u = 0; u < AD_UNROLL; ++u) kk[u] = *reinterpret_cast<const Vec*>(st + min(s0 + u * GROUPS, count - 1) * C::ROW);
#pragma unroll
      for (int u = 0; u < AD_UNROLL; ++u) vv[u] = *reinterpret_cast<const Vec*>(st + C::HALF + min(s0 + u * GROUPS, count - 1) * C::ROW);
      float dot[AD_UNROLL];
#pragma unroll
      for (int u = 0; u < AD_UNROLL; ++u) {
        float d = 0.f;
#pragma unroll
        for (int e = 0; e < 8; ++e) d += q[e] * xl_to_float(kk[u].v[e]);
        dot[u] = d;
      }
      // four sums over the lanes of a group by halving: of its quarters the first ends up with dot[0], ...
      const bool upper = lane & (LANES / 2), odd = lane & (LANES / 4);
      float d0 = (upper ? dot[2] : dot[0]) + __shfl_xor_sync(0xffffffffu, upper ? dot[0] : dot[2], LANES / 2);
      float d1 = (upper ? dot[3] : dot[1]) + __shfl_xor_sync(0xffffffffu, upper ? dot[1] : dot[3], LANES / 2);
      d0 = (odd ? d1 : d0) + __shfl_xor_sync(0xffffffffu, odd ? d0 : d1, LANES / 4);
#pragma unroll
      for (int off = LANES / 8; off > 0; off >>= 1) d0 += __shfl_xor_sync(0xffffffffu, d0, off);
      float m_new = m;
#pragma unroll
      for (int u = 0; u < AD_UNROLL; ++u) {
        dot[u] = __shfl_sync(0xffffffffu, d0, group * LANES + u * (LANES / 4));
        if (s0 + u * GROUPS >= count) dot[u] = -INFINITY;
        m_new = fmaxf(m_new, dot[u]);
      }
      const float top = m_new == -INFINITY ? 0.f : m_new;  // a group may have none of the positions yet
      const float corr = __expf(m - top);
      l *= corr;
#pragma unroll
      for (int e = 0; e < 8; ++e) o[e] *= corr;
#pragma unroll
      for (int u = 0; u < AD_UNROLL; ++u) {
        const float w = __expf(dot[u] - top);  // exp(-inf) = 0 for the masked duplicates
        l += w;
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] += w * xl_to_float(vv[u].v[e]);
      }
      m = m_new;
    }
    mbar_arrive_reads_done(&empty_bar[stage]);
    if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
  }
  // merge the groups of this CTA, a thread per feature
  const int stream = warp * GROUPS + group;
  if (at_d == 0) { sm[stream] = m; sl[stream] = l; }
  *reinterpret_cast<float4*>(&so[stream][at_d]) = make_float4(o[0], o[1], o[2], o[3]);
  *reinterpret_cast<float4*>(&so[stream][at_d + 4]) = make_float4(o[4], o[5], o[6], o[7]);
  ad_sync<W>();
  T* out = (T*)p.out + (long long)b * p.ldo + h * D;
  float* mine = p.part + ((long long)bh * splits + split) * (D + 2);
  for (int d = threadIdx.x; d < D; d += W * 32) {
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < STREAMS; ++w) mm = fmaxf(mm, sm[w]);
    float ll = 0.f, acc = 0.f;
#pragma unroll
    for (int w = 0; w < STREAMS; ++w) {
      const float f = (sm[w] == -INFINITY) ? 0.f : __expf(sm[w] - mm);
      ll += sl[w] * f;
      acc += so[w][d] * f;
    }
    if (splits == 1) {
      out[d] = xl_from_float<T>(acc / ll);
    } else {
      if (d == 0) { mine[0] = mm; mine[1] = ll; }
      mine[2 + d] = acc;
    }
  }
  if (splits == 1) return;
  ad_sync<W>();
  if (threadIdx.x == 0) {
    __threadfence();  // for the stores of all, which the barrier has ordered before it
    is_last = atomicAdd(p.counters + bh, 1u) == (unsigned int)splits - 1;
  }
  ad_sync<W>();
  if (!is_last) return;
  __threadfence();
  const float* part = p.part + (long long)bh * splits * (D + 2);
  for (int d = threadIdx.x; d < D; d += W * 32) {
    float mm = -INFINITY;
#pragma unroll 8
    for (int s = 0; s < splits; ++s) mm = fmaxf(mm, __ldcg(part + s * (D + 2)));
    float ll = 0.f, acc = 0.f;
#pragma unroll 8
    for (int s = 0; s < splits; ++s) {
      const float* ps = part + s * (D + 2);
      const float ms = __ldcg(ps), f = ms == -INFINITY ? 0.f : __expf(ms - mm);
      ll += __ldcg(ps + 1) * f;
      acc += __ldcg(ps + 2 + d) * f;
    }
    out[d] = xl_from_float<T>(acc / ll);
  }
  if (threadIdx.x == 0) p.counters[bh] = 0;
}

template <typename T, int D, int W> int ad_launch(const AdParams& p, int BH, int splits, cudaStream_t s) {
  using C = AdCfg<D, W>;
  static XlPerDevice smem;
  XL_TRY(xl_allow_smem(attn_decode_kernel<T, D, W>, C::SMEM, smem));
  const cudaError_t e = xl_launch_overlapped(attn_decode_kernel<T, D, W>, dim3(BH, splits), dim3(C::THREADS), (size_t)C::SMEM, s, p);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}
template <typename T, int W> int ad_pick(const AdParams& p, int BH, int D, int splits, cudaStream_t s) {
  return D == 256 ? ad_launch<T, 256, W>(p, BH, splits, s)
                  : (D == 128 ? ad_launch<T, 128, W>(p, BH, splits, s) : ad_launch<T, 64, W>(p, BH, splits, s));
}
template <typename T> int ad_warps(const AdParams& p, int BH, int D, int splits, int warps, cudaStream_t s) {
  return warps == 8 ? ad_pick<T, 8>(p, BH, D, splits, s) : (warps == 4 ? ad_pick<T, 4>(p, BH, D, splits, s) : ad_pick<T, 2>(p, BH, D, splits, s));
}

}  // namespace

// qkv: rows of ldq elements, q first (H * D of them; with `append` k and v behind it); out: rows of ldo elements (H * D written), which
// may be the rows' v part. Caches (B, H, Smax, D) of 16-byte aligned rows. append: q and k are rotated (first R features of each head,
// interleaved pairs, tables (Smax, R / 2) of the type of qkv; qkv itself stays) for position *pos_ptr, k and v written to the caches there;
// else the cache holds position *pos_ptr already. scratch: B * H * splits * (D + 2) floats; counters: B * H zero-initialised words (left
// zeroed); both only for splits > 1. warps: 2, 4 or 8 per CTA. D in {64, 128, 256}; ldq, ldo multiples of 8. read_ahead: *pos_ptr and the caches were complete before
// the previous launch on the stream. Returns -1 for arguments it does not take.
XL_API int xl_attn_decode(const void* qkv, long long ldq, const void* sin_t, const void* cos_t, void* k_cache, void* v_cache, void* out,
                          long long ldo, float* scratch, unsigned int* counters, const int* pos_ptr, int B, int H, int D, int R,
                          int Smax, float scale, int splits, int warps, int append, int read_ahead, int dtype, int* err, cudaStream_t s) {
  if ((D != 64 && D != 128 && D != 256) || (warps != 2 && warps != 4 && warps != 8) || splits < 1 || splits > 65535 || dtype == XL_F32 || (ldq % 8) || (ldo % 8)) return -1;
  if (splits > 1 && (scratch == nullptr || counters == nullptr)) return -1;
  if (append && (R < 0 || (R & 1) || R > D || (R && (!sin_t || !cos_t)))) return -1;
  if (((uintptr_t)qkv | (uintptr_t)k_cache | (uintptr_t)v_cache) & 15) return -1;
  const AdParams p{qkv, ldq, k_cache, v_cache, out, ldo, scratch, counters, pos_ptr, sin_t, cos_t, H, Smax, R, append, read_ahead, scale, err};
  return dtype == XL_BF16 ? ad_warps<__nv_bfloat16>(p, B * H, D, splits, warps, s) : ad_warps<__half>(p, B * H, D, splits, warps, s);
}
