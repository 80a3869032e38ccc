// Edge pruning + task/slice layout (K5), init normalisation (K6) and the Hogwild SGD epoch
// (K7).
//
// Layout.  The kept edges of the symmetric graph are grouped by head row and cut into tasks
// of at most `chunk` edges (see SgdLayout), packed 32 to a slice; the head row's live embedding
// is kept in registers while its task runs.  A slice's entries are lane major: task l's entries
// are contiguous at base + l * width (width = the slice's longest task rounded up to 4 entries,
// padding never fires).  In DRAM-bound layouts entry e of task l sits at base + 32 e + l instead,
// so a warp's loads cover whole 256-byte rows (see pick_epoch_kernel).  The reference writes a
// head row only from edges whose head it is (optimize_layout_euclidean.rs:281-306, :338),
// so a task that is a whole row reproduces the reference's sequential per-row order with
// no lost head updates; the rare long rows (kNN hubs) are split so that one row cannot
// serialise an epoch, and each partial task merges its head delta with an atomic add.
// Tail moves (fire-and-forget atomic adds, see sub_row) and negative samples (racy loads)
// touch the per-call snapshot buffer, where the reference reads and writes it racily.
//
// Schedule.  The reference keeps four f64 arrays per edge (optimizer.rs:33-43).  Here one
// u32 per edge holds Q = ceil(2^32 / epochs_per_sample) and the state is recomputed in
// exact integer arithmetic: the edge has fired m(n) = (n*Q) >> 32 times by epoch n, so it
// fires at n iff m(n) > m(n-1) (at most once per epoch, never at epoch 0; :277, :308), and
// a firing with index m draws y(n) - y(p) negatives, y(x) = (x*neg*Q) >> 32 and p the epoch
// of firing m-1 (y(n) - 1 for the first firing): the closed form of :310-311 / :343.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <utility>
#include <vector>

#include "ub_internal.hpp"
#include "umma.cuh"

namespace ub {
namespace {

constexpr uint32_t PAD_ROW = 0xFFFFFFFFu;

// DRAM-bound layouts (sgd_epoch_dram): 12 negative rows fetched together, 3 blocks per SM.  Their
// random row loads go to DRAM and their warps are limited by registers either way, so more loads
// in flight per lane beat more warps (30 epochs of a 20M-point roll: 8 / 4: 310.8 ms, 10 / 3:
// 295.1, 12 / 3: 295.2, 12 / 2: 313.4, 16 / 2: 316.0, 24 / 2: 317.7; 40M points, 24 epochs:
// 8 / 4: 590.4, 12 / 3: 562.6, 16 / 2: 564.9).
constexpr int NB_DRAM = 12, MINB_DRAM = 3;
// The lane kernel (sgd_epoch_kernel2) comes in two register budgets.  Large graphs (many waves of
// warps): 4 negative rows fetched together and 5 resident 256-thread blocks per SM.  Graphs that
// fill about two waves or fewer are bound by the chain of dependent loads of their busiest lanes: 8
// negative rows fetched together and 4 blocks per SM.  (2M points, 500 epochs, SGD ms: 4 / 5 314.0, 8 / 4
// 317.6, 6 / 4 330.9, 4 / 4 343.5.)
constexpr int NB_WIDE = 4, MINB_WIDE = 5;
constexpr int NB_SHORT = 8, MINB_SHORT = 4;
// The pooled kernel: 8 negative rows fetched together, 8 blocks of 128 threads per SM (64
// registers).  2M points, us per epoch: 8 / 8: 482, 6 / 8: 480, 6 / 9: 481, 4 / 10: 516, 4 / 8: 511;
// 300k points: 92, 98, 98, 106, 106.
constexpr int POOL_BT = 128, NB_POOL = 8, MINB_POOL = 8;

// ------------------------------------------------------------------------------ negatives' RNG
// Counter-based: the firing of entry `idx` at `epoch` draws its negatives in pairs; pair t is
// the SplitMix64 finaliser (Steele, Lea, Flood, "Fast splittable pseudorandom number
// generators", OOPSLA 2014) of a counter derived from (seed, idx, epoch, t), and each 32-bit
// half maps to [0, n) by a multiply-high.  The reference draws from an unseeded thread-local
// generator (optimize_layout_euclidean.rs:314), so parity with it is statistical.
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
struct NegRng {
  uint64_t base;
  __device__ __forceinline__ NegRng(uint64_t seed, uint64_t idx, uint32_t epoch)
      : base(seed ^ (idx * 0x9E3779B97F4A7C15ull) ^ ((uint64_t)epoch * 0xC2B2AE3D27D4EB4Full)) {}
  __device__ __forceinline__ uint64_t pair(uint32_t t) const { return mix64(base + (uint64_t)t * 0xD1B54A32D192ED03ull); }
};

// ------------------------------------------------------------------------------ schedule
__host__ __device__ __forceinline__ uint32_t q_minus_1(double eps) {
  if (!(eps > 0.0)) return 0u;
  const double x = ceil(4294967296.0 / eps);
  if (x >= 4294967296.0) return 0xFFFFFFFFu;
  if (x < 1.0) return 0u;
  return (uint32_t)x - 1u;
}
// All schedule helpers take q = Q - 1 (the stored u32).  n*Q = n*q + n fits in 64 bits for
// any u32 n, and the product is a single 32x32->64 multiply.
__device__ __forceinline__ uint64_t fires_by(uint32_t n, uint32_t q) {
  return ((uint64_t)n * q + n) >> 32;
}
// Smallest epoch x with fires_by(x) >= m.
__device__ __forceinline__ uint32_t fire_epoch(uint64_t m, uint32_t q) {
  const float est = (float)m * __fdividef(4294967296.0f, (float)q + 1.0f);
  uint32_t x = est > 0.0f ? (est < 4294967040.0f ? (uint32_t)ceilf(est) : 0xFFFFFF00u) : 0u;
  for (int t = 0; t < 8 && x > 0 && fires_by(x - 1, q) >= m; ++t) --x;
  for (int t = 0; t < 8 && fires_by(x, q) < m; ++t) ++x;
  return x;
}

// Negatives drawn in total after m firings.
__device__ __forceinline__ uint64_t negatives_after(uint64_t m, uint32_t q, uint32_t neg) {
  if (m == 0) return 0;
  const int64_t t = (int64_t)fires_by(fire_epoch(m, q) * neg, q) - 1;
  return t > 0 ? (uint64_t)t : 0ull;
}
// Fires at epoch n iff fires_by(n) > fires_by(n - 1), i.e. iff the low 32 bits of (n - 1) * Q
// are at least 2^32 - Q (Q <= 2^32, so the count grows by at most one): one 32-bit multiply.
__device__ __forceinline__ bool fires_at(uint32_t n, uint32_t q) {
  const uint32_t nm1 = n - 1u;
  return n > 0 && nm1 * q + nm1 >= ~q;
}
// Negatives drawn by the firing at epoch n (n * neg < 2^32 is checked on the host):
// y(n) - y(p) with y(x) = fires_by(x * neg) and p the epoch of the previous firing, or
// y(n) - 1 for the first.  With n Q = m 2^32 + f (0 <= f < Q, as it fires at n) the previous firing
// is t = floor((2^32 + f) / Q) epochs back and p Q = (m - 1) 2^32 + g, g = (2^32 + f) - t Q, so
// y(n) = m neg + floor(neg f / 2^32) and y(p) = (m - 1) neg + floor(neg g / 2^32).  t <= n <
// MAX_EPOCHS = 2^21 (checked on the host), so the float quotient is within one of it and g's sign
// and size correct it.
__device__ __forceinline__ uint32_t negatives_at(uint32_t n, uint32_t q, uint32_t neg) {
  const uint64_t nq = (uint64_t)n * q + n, Q = (uint64_t)q + 1;
  const uint32_t f = (uint32_t)nq, m = (uint32_t)(nq >> 32);
  const int64_t span = (int64_t)(((uint64_t)1 << 32) + f);
  const uint32_t t = (uint32_t)__fdividef(4294967296.0f + (float)f, (float)Q);
  int64_t g = span - (int64_t)((uint64_t)t * Q);
  if (g < 0) g += (int64_t)Q;
  else if (g >= (int64_t)Q) g -= (int64_t)Q;
  const uint32_t upto = __umulhi(neg, f);
  const int32_t d = (int32_t)(neg + upto - (m > 1 ? __umulhi(neg, (uint32_t)g) : 1u));
  return d > 0 ? (uint32_t)d : 0u;
}

// Two-lane FP32 arithmetic on a 2-D row (each lane the same IEEE operation as the scalar one).
__device__ __forceinline__ uint64_t pk2(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(__float_as_uint(x)), "r"(__float_as_uint(y)));
  return r;
}
__device__ __forceinline__ void up2(uint64_t v, float& x, float& y) {
  uint32_t a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(v));
  x = __uint_as_float(a);
  y = __uint_as_float(b);
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// ------------------------------------------------------------------------------ K7

template <int DIM>
__device__ __forceinline__ void load_row(float (&v)[DIM], const float* p) {
  if constexpr (DIM == 2) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = t.x;
    v[1] = t.y;
  } else if constexpr (DIM == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else {
#pragma unroll
    for (int d = 0; d < DIM; ++d) v[d] = p[d];
  }
}
// The same through L2 only.
template <int DIM>
__device__ __forceinline__ void load_row_l2(float (&v)[DIM], const float* p) {
  if constexpr (DIM == 2) {
    const float2 t = __ldcg(reinterpret_cast<const float2*>(p));
    v[0] = t.x;
    v[1] = t.y;
  } else if constexpr (DIM == 4) {
    const float4 t = __ldcg(reinterpret_cast<const float4*>(p));
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else {
#pragma unroll
    for (int d = 0; d < DIM; ++d) v[d] = __ldcg(p + d);
  }
}
template <int DIM>
__device__ __forceinline__ void store_row(float* p, const float (&v)[DIM]) {
  if constexpr (DIM == 2) {
    *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  } else if constexpr (DIM == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  } else {
#pragma unroll
    for (int d = 0; d < DIM; ++d) p[d] = v[d];
  }
}

// Tail move (optimize_layout_euclidean.rs:303-305) as a fire-and-forget atomic add.  The
// reference's racy read-modify-write rarely collides on a CPU (a vertex's few tail moves per
// epoch come from rows processed at different times); with every row of an epoch in flight
// at once, plain stores would drop most of them, so the add is atomic to keep the
// reference's statistics.
template <int DIM>
__device__ __forceinline__ void sub_row(float* p, const float (&g)[DIM]) {
  if constexpr (DIM == 2) {
    atomicAdd(reinterpret_cast<float2*>(p), make_float2(-g[0], -g[1]));
  } else if constexpr (DIM == 4) {
    atomicAdd(reinterpret_cast<float4*>(p), make_float4(-g[0], -g[1], -g[2], -g[3]));
  } else {
#pragma unroll
    for (int d = 0; d < DIM; ++d) atomicAdd(p + d, -g[d]);
  }
}

// Force law of the generic-metric path (layout/optimize_layout_generic.rs:65-119) with the
// built-in output metric EuclideanMetric (distances.rs:22-37): distance d = sqrt(sum diff^2),
// gradient diff / (d + 1e-6), w = 1 / (1 + a d^(2b)).  Returns the coefficient c that
// multiplies the gradient: 2b (w - 1) / (d + 1e-6) for an attraction, 2 gamma b w / (d + 1e-6)
// for a repulsion (`scale` = 2b or 2 gamma b, `bias` = -1 or 0); *den receives d + 1e-6.
__device__ __forceinline__ float metric_coeff(float ds, float a, float two_b, float scale, float bias,
                                              float* den) {
  const float dist = sqrtf(ds);
  *den = dist + 1e-6f;
  const float w = dist > 0.0f ? 1.0f / (1.0f + a * __powf(dist, two_b)) : 1.0f;
  return __fdividef(scale * (w + bias), *den);
}

// The Euclidean rule's step of a head row (optimize_layout_euclidean.rs:284-306, :319-339) with
// the shortest chain from the row to its update, which is what a task's firings wait for: the
// squared distance carries the smallest normal number along (a subnormal one would cost scaling
// instructions around each approximate log2 / exp2 / reciprocal), ds^b = 2^(b log2 ds), and the
// denominators are one fused step behind it.  Like the rule, an attraction at distance 0 or NaN has
// coefficient 0 and a repulsion moves only where its coefficient is above 0 (it is 0 at an infinite
// distance): a row with a NaN or infinite coordinate leaves those that draw it alone.
__device__ __forceinline__ float ftz_log2(float x) { float r; asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float ftz_exp2(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float ftz_rcp(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
// Rust f32::clamp(-4, 4) (utils/clip.rs:13-15): NaN passes through.
__device__ __forceinline__ float clip4(float v) {
  float r;
  asm("min.NaN.f32 %0, %1, 0f40800000;" : "=f"(r) : "f"(v));
  asm("max.NaN.f32 %0, %1, 0fC0800000;" : "=f"(r) : "f"(r));
  return r;
}
template <int DIM>
__device__ __forceinline__ float square_ftz(const float (&df)[DIM]) {
  float ds = FLT_MIN;
#pragma unroll
  for (int d = 0; d < DIM; ++d) ds = fmaf(df[d], df[d], ds);
  return ds;
}
// Attractive move g of the head row (the tail gets -g): coefficient -2ab ds^b / (ds (a ds^b ds + 1)).  What keeps
// the rule's limits stands beside the chain from the distance to the reciprocal: a NaN distance counts as 0,
// whose coefficient is 0, and where the denominator overflows the row's difference is left out of the
// product, which could overflow before the reciprocal's 0 meets it.
template <int DIM>
__device__ __forceinline__ void attract(float (&cur)[DIM], const float (&o)[DIM], float (&g)[DIM], const SgdParams& p,
                                        float alpha) {
  float df[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) df[d] = cur[d] - o[d];
  const float sq = square_ftz<DIM>(df), ds = fmaxf(sq, FLT_MIN);
  const float pb = ftz_exp2(p.b * ftz_log2(ds)), den = fmaf(p.a * ds * ds, pb, ds), inv = ftz_rcp(den);
  const float num = sq > FLT_MIN ? p.neg_attr * pb : 0.0f;
  const bool far = !(den <= FLT_MAX);
#pragma unroll
  for (int d = 0; d < DIM; ++d) g[d] = clip4((num * (far ? 0.0f : df[d])) * inv) * alpha;
}
// Repulsive move from row o: coefficient 2 gamma b / ((0.001 + ds)(a ds^b ds + 1)), where it is above 0; the
// denominator's range tells beside its reciprocal.  `rep` = max(2 gamma b, 0).
template <int DIM>
__device__ __forceinline__ bool repel_move(const float (&df)[DIM], float (&g)[DIM], const SgdParams& p, float rep) {
  const float ds = square_ftz<DIM>(df), u = 0.001f + ds, v = u * (p.a * ds);
  const float den = fmaf(v, ftz_exp2(p.b * ftz_log2(ds)), u), inv = ftz_rcp(den);
#pragma unroll
  for (int d = 0; d < DIM; ++d) g[d] = clip4((rep * df[d]) * inv);
  return den > 0.0f && den <= FLT_MAX;
}
template <int DIM>
__device__ __forceinline__ void repel(float (&cur)[DIM], const float (&o)[DIM], const SgdParams& p, float rep, float alpha) {
  float df[DIM], g[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) df[d] = cur[d] - o[d];
  if (repel_move<DIM>(df, g, p, rep)) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) cur[d] = fmaf(g[d], alpha, cur[d]);
  }
}

// One fired edge (optimize_layout_euclidean.rs:278-343, or with GEN the generic-metric rule
// of optimize_layout_generic.rs:57-121): attractive step on (head, tail), then `nneg`
// negative samples, all reading the snapshot buffer.  The tail row and a batch of negative
// rows are fetched together before the (sequential) updates of `cur`.  FUSED takes the Euclidean rule's moves from
// attract / repel above; without it every operation stands by itself.
template <int DIM, bool GEN, int NEG_BATCH, bool FUSED>
__device__ __forceinline__ void fired_edge(float (&cur)[DIM], uint32_t r, uint32_t k, uint32_t nneg,
                                           float* snap, const SgdParams& p, float alpha, uint64_t idx,
                                           uint32_t epoch, uint32_t seg_lo, uint32_t seg_n) {
  const float a = p.a, b = p.b, rep = fmaxf(p.pos_rep, 0.0f);
  float* oth = snap + (uint64_t)k * DIM;
  float o[DIM];
  load_row<DIM>(o, oth);
  // Negative q uses half (q & 1) of pair (q >> 1) for this (entry, epoch).
  uint32_t kk[NEG_BATCH];
  float ob[NEG_BATCH][DIM];
  const NegRng rng(p.seed, idx, epoch);
  uint64_t rnd = 0;
  uint32_t rpair = 0xFFFFFFFFu;
  auto fetch = [&](uint32_t q0) {
#pragma unroll
    for (int q = 0; q < NEG_BATCH; ++q) {
      const uint32_t qq = q0 + q;
      if (qq < nneg) {
        if ((qq >> 1) != rpair) {
          rpair = qq >> 1;
          rnd = rng.pair(rpair);
        }
        const uint32_t rv = (qq & 1) ? (uint32_t)(rnd >> 32) : (uint32_t)rnd;
        kk[q] = seg_lo + __umulhi(rv, seg_n);
        if constexpr (DIM == 2) {
          // uniform rows, rarely reused by this SM: cached in L2 only, so they do not evict
          // the tail and head lines L1 serves (2M workload, 500 epochs: 311.1-311.2 against
          // 311.8-311.9 ms; renamed 20M roll, 30 epochs: 219.7-220.1 against 221.3-223.6 ms)
          const float2 t = __ldcg(reinterpret_cast<const float2*>(snap + (uint64_t)kk[q] * DIM));
          ob[q][0] = t.x;
          ob[q][1] = t.y;
        } else {
          load_row<DIM>(ob[q], snap + (uint64_t)kk[q] * DIM);
        }
      }
    }
  };
  fetch(0);
  // attractive step (:284-306)
  float ds = 0.0f;
#pragma unroll
  for (int d = 0; d < DIM; ++d) { const float df = cur[d] - o[d]; ds += df * df; }
  float g[DIM];
  if constexpr (FUSED) {
    attract<DIM>(cur, o, g, p, alpha);
#pragma unroll
    for (int d = 0; d < DIM; ++d) cur[d] += g[d];
  } else if constexpr (GEN) {
    // head += clip(c * grad) alpha; tail += clip(c * rev_grad) alpha with rev_grad = -grad
    float den;
    const float gc = metric_coeff(ds, a, p.two_b, p.two_b, -1.0f, &den);
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      g[d] = clip4(gc * __fdividef(cur[d] - o[d], den)) * alpha;
      cur[d] += g[d];
    }
  } else {
    float gc = 0.0f;
    if (ds > 0.0f) {
      const float pb = __powf(ds, b);
      gc = __fdividef(p.neg_attr * pb, ds * (a * pb * ds + 1.0f));
    }
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      g[d] = clip4(gc * (cur[d] - o[d])) * alpha;
      cur[d] += g[d];
    }
  }
  sub_row<DIM>(oth, g);
  // negative samples (:313-341)
  for (uint32_t q0 = 0; q0 < nneg; q0 += NEG_BATCH) {
    if (q0 > 0) fetch(q0);  // more than NEG_BATCH negatives in this firing
#pragma unroll
    for (int q = 0; q < NEG_BATCH; ++q) {
      if (q0 + q >= nneg) break;
      if (kk[q] == r) continue;
      if constexpr (FUSED) {
        repel<DIM>(cur, ob[q], p, rep, alpha);
        continue;
      }
      if constexpr (DIM == 2 && !GEN) {
        // the same operations as the generic-DIM code below, two columns per instruction
        const uint64_t c2 = pk2(cur[0], cur[1]);
        const uint64_t df2 = sub2(c2, pk2(ob[q][0], ob[q][1]));
        float df0, df1;
        up2(df2, df0, df1);
        const float dsn = df0 * df0 + df1 * df1;
        float gr = 0.0f;
        if (dsn > 0.0f) {
          const float pb = __powf(dsn, b);
          gr = __fdividef(p.pos_rep, (0.001f + dsn) * (a * pb * dsn + 1.0f));
        }
        if (gr > 0.0f) {
          float t0, t1;
          up2(mul2(pk2(gr, gr), df2), t0, t1);
          up2(fma2(pk2(clip4(t0), clip4(t1)), pk2(alpha, alpha), c2), cur[0], cur[1]);
        }
        continue;
      }
      float dsn = 0.0f;
#pragma unroll
      for (int d = 0; d < DIM; ++d) { const float df = cur[d] - ob[q][d]; dsn += df * df; }
      if constexpr (GEN) {
        float den;
        const float gr = metric_coeff(dsn, a, p.two_b, p.pos_rep, 0.0f, &den);
#pragma unroll
        for (int d = 0; d < DIM; ++d) cur[d] += clip4(gr * __fdividef(cur[d] - ob[q][d], den)) * alpha;
      } else {
        float gr = 0.0f;
        if (dsn > 0.0f) {
          const float pb = __powf(dsn, b);
          gr = __fdividef(p.pos_rep, (0.001f + dsn) * (a * pb * dsn + 1.0f));
        }
        if (gr > 0.0f) {
#pragma unroll
          for (int d = 0; d < DIM; ++d) cur[d] += clip4(gr * (cur[d] - ob[q][d])) * alpha;
        }
      }
    }
  }
}

// A lane per task with independent progress: each lane walks its own task through a small register
// window of entries (refilled on demand, 4 loads in flight), so a warp runs as long as its busiest
// task rather than its busiest lane of every batch.  Its order of updates is the one that layouts
// at small learning rates keep (see pick_epoch_kernel).
template <int DIM, bool GEN, int NEG_BATCH, int MINB, bool LM, bool SEG>
__global__ void __launch_bounds__(256, MINB) sgd_epoch_kernel2(
    const uint64_t* __restrict__ slice_base, const uint32_t* __restrict__ slice_width,
    const uint32_t* __restrict__ split_mask, const uint32_t* __restrict__ rowid,
    const uint2* __restrict__ entry, uint64_t n_slices, float* __restrict__ live, float* snap,
    SgdParams p, uint32_t epoch, float alpha) {
  constexpr int W = 4;
  const uint64_t slice = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  if (slice >= n_slices) return;
  const uint32_t r = rowid[slice * 32 + lane];
  const bool active = r != PAD_ROW;
  const uint32_t width = active ? slice_width[slice] : 0u;
  const uint64_t base = slice_base[slice];
  const bool split = (split_mask[slice] >> lane) & 1u;
  uint32_t seg_lo = 0, seg_n = p.n_vertices;
  if constexpr (SEG) {
    if (active) {
      const uint32_t sg = p.row_seg[r];
      seg_lo = (uint32_t)p.seg_off[sg];
      seg_n = (uint32_t)(p.seg_off[sg + 1] - p.seg_off[sg]);
    }
  }
  float cur[DIM], start[DIM];
  float* hrow = live + (uint64_t)(active ? r : 0) * DIM;
  if (active) load_row<DIM>(cur, hrow);
  else
#pragma unroll
    for (int d = 0; d < DIM; ++d) cur[d] = 0.0f;
#pragma unroll
  for (int d = 0; d < DIM; ++d) start[d] = cur[d];
  const uint32_t n = epoch;
  static_assert(W % 4 == 0, "windows are whole 4-entry sectors");
  // this lane's entries: contiguous (lane major) or every 32nd (interleaved)
  const uint2* lent = LM ? entry + base + (uint64_t)lane * width : entry + base + lane;
  uint2 win[W];
  uint32_t mask = 0, ew = 0, ebase = 0;
  for (;;) {
    while (mask == 0 && ew < width) {
      ebase = ew;
      if (LM) {
        // width is a multiple of W (slice_meta_kernel): the window lies inside the lane's entries
#pragma unroll
        for (int j = 0; j < W; j += 2) {
          const uint4 v = __ldg(reinterpret_cast<const uint4*>(lent + ew + j));
          win[j] = make_uint2(v.x, v.y);
          win[j + 1] = make_uint2(v.z, v.w);
        }
      } else {
#pragma unroll
        for (int j = 0; j < W; ++j) {
          const uint32_t e = ew + j;
          win[j] = e < width ? __ldg(lent + (uint64_t)e * 32) : make_uint2(0u, 0u);
        }
      }
#pragma unroll
      for (int j = 0; j < W; ++j)
        if (fires_at(n, win[j].y)) mask |= 1u << j;
      ew += W;
    }
    if (!__any_sync(0xFFFFFFFFu, mask != 0)) break;
    if (mask) {
      const int j = __ffs(mask) - 1;
      mask &= mask - 1;
      uint2 en = win[0];
#pragma unroll
      for (int t = 1; t < W; ++t)
        if (t == j) en = win[t];
      const uint32_t nneg = negatives_at(n, en.y, p.neg_rate);
      const uint64_t idx = LM ? base + (uint64_t)lane * width + ebase + j : base + (uint64_t)(ebase + j) * 32 + lane;
      fired_edge<DIM, GEN, NEG_BATCH, false>(cur, r, en.x, nneg, snap, p, alpha, idx, epoch, seg_lo, seg_n);
    }
  }
  if (active) {
    if (split) {
#pragma unroll
      for (int d = 0; d < DIM; ++d) atomicAdd(hrow + d, cur[d] - start[d]);
    } else {
      store_row<DIM>(hrow, cur);
    }
  }
}

// DRAM-bound layouts (1-D and 2-D, interleaved entries): a lane per task with independent progress -
// each lane finds the firings of 16 of its entries at a time and walks them - so a warp runs as
// long as its busiest task.  (A 4-entry window held in registers, refilled about once per firing,
// took 5M-point epochs from 1,156 to 1,530 us.)
constexpr int DRAM_WIN = 16;
template <int DIM>
__global__ void __launch_bounds__(256, MINB_DRAM) sgd_epoch_dram(
    const uint64_t* __restrict__ slice_base, const uint32_t* __restrict__ slice_width,
    const uint32_t* __restrict__ split_mask, const uint32_t* __restrict__ rowid,
    const uint2* __restrict__ entry, uint64_t n_slices, float* __restrict__ live, float* snap,
    SgdParams p, uint32_t epoch, float alpha) {
  const uint64_t slice = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  if (slice >= n_slices) return;
  const uint32_t r = rowid[slice * 32 + lane];
  const bool active = r != PAD_ROW;
  const uint32_t width = active ? slice_width[slice] : 0u;
  const uint64_t first = slice_base[slice] + lane;
  const bool split = (split_mask[slice] >> lane) & 1u;
  float cur[DIM], start[DIM];
  float* hrow = live + (uint64_t)(active ? r : 0) * DIM;
  load_row<DIM>(cur, hrow);
#pragma unroll
  for (int d = 0; d < DIM; ++d) start[d] = cur[d];
  const uint2* lent = entry + first;
  uint32_t mask = 0, ew = 0, ebase = 0;
  uint2 nx = make_uint2(0u, 0u);  // the next fired entry
  for (;;) {
    if (mask == 0) {
      while (mask == 0 && ew < width) {
        ebase = ew;
#pragma unroll
        for (int j = 0; j < DRAM_WIN; ++j) {
          const uint32_t q = ew + j < width ? __ldg(&lent[(uint64_t)(ew + j) * 32].y) : 0u;
          mask |= fires_at(epoch, q) ? 1u << j : 0u;
        }
        ew += DRAM_WIN;
      }
      if (mask) nx = __ldg(lent + (uint64_t)(ebase + __ffs(mask) - 1) * 32);
    }
    if (!__any_sync(0xFFFFFFFFu, mask != 0)) break;
    if (mask) {
      const uint2 en = nx;
      const uint64_t idx = first + (uint64_t)(ebase + __ffs(mask) - 1) * 32;
      mask &= mask - 1;
      if (mask) nx = __ldg(lent + (uint64_t)(ebase + __ffs(mask) - 1) * 32);
      fired_edge<DIM, false, NB_DRAM, true>(cur, r, en.x, negatives_at(epoch, en.y, p.neg_rate), snap, p, alpha, idx, epoch,
                                      0u, p.n_vertices);
    }
  }
  if (active) {
    if (split) {
#pragma unroll
      for (int d = 0; d < DIM; ++d) atomicAdd(hrow + d, cur[d] - start[d]);
    } else {
      store_row<DIM>(hrow, cur);
    }
  }
}

// The epoch of L2-resident layouts: a block of POOL_BT threads takes as many tasks.  For every
// window of 32 entries it (1) evaluates the schedule of all its tasks' entries, 8 lanes reading 64
// consecutive bytes of a task, which leaves one bit per entry, (2) sorts the tasks that fire by
// their number of firings (counting sort, descending), and (3) gives thread i the i-th of them.
// What bounds it: the random rows - per firing a tail, its atomic add and about 5 negatives, one
// 32-byte L2 sector each.  Such a mix runs at most at 260 G/s here whatever the path (plain,
// L2-only, asynchronous copies), 0.385 ms of the 2M-point epoch.  A warp whose lanes own fixed tasks
// has half of them idle (its tasks' firings differ from epoch to epoch), and reading the schedule in
// per-lane windows cost a quarter more requests: 2M points 537 -> 474 us per epoch, 300k 102 -> 92,
// 70k 39 -> 34.  Larger pools (256 or 512 tasks, warps taking 32 at a time from the sorted list)
// were slower: a block's heavy warps outlast the others, 727 / 945 us at 2M.
// Small graphs are bound by the chain of one task's firings - row loads, then 6 dependent updates -
// with the chip half empty.  Drawing a firing's rows during the loads of the one before took the
// generator out of it (500 points 18.6 -> 14.3 us per epoch, 10k 21.3 -> 17.5, 70k 31.0 -> 28.4, 2M
// 456 -> 439, in 100 epochs at small rates).  At rate 1, this kernel / a lane per task, us per epoch: 500
// points 15.5 / 30.6, 10k 17.5 / 31.5, 70k 28.6 / 39.2, 300k 83 / 106, 1M 236 / 305, 2M 463 / 582 (495 on
// average over 500 epochs, at the power limit).  Loading the rows themselves one firing ahead, with
// 8 lanes per task, ran 500 points in 11 us and no larger set faster than this, but its updates
// see older rows, and layouts of some thousand points moved by more than two runs differ.
// MANY: rates whose firings draw more negatives than are fetched together (NB_POOL or more a sample) fetch them as many
// at a time, too, and draw the next firing's rows after that (20k points, 60 epochs, 20 / 50 negatives a sample:
// 7.5 / 17.2 ms a fit with one row after another, 4.4 / 8.2 so, a lane per task 6.6 / 13.5).  Lower rates lose by the
// later draw (us per epoch without / with, 20k points: 5 a sample 18.8 / 19.6, 7 29.6 / 28.8, 8 36.4 / 31.4;
// 300k: 79.6 / 80.1, 100.2 / 103.1, 116.4 / 116.4).
// `early` lets the next epoch's blocks start as soon as this launch's last ones have, otherwise at
// its end (see sgd_epoch).
constexpr int POOL_WIN = 32;
template <int DIM, bool GEN, bool SEG, bool MANY>
__global__ void __launch_bounds__(POOL_BT, MINB_POOL) sgd_epoch_pool(
    const uint64_t* __restrict__ slice_base, const uint32_t* __restrict__ slice_width,
    const uint32_t* __restrict__ split_mask, const uint32_t* __restrict__ rowid,
    const uint2* __restrict__ entry, uint64_t n_slices, float* __restrict__ live, float* snap,
    SgdParams p, uint32_t epoch, float alpha, bool early) {
  const float rep = fmaxf(p.pos_rep, 0.0f);
  constexpr int SL = POOL_BT / 32;  // slices: one per warp while the schedule is evaluated
  // Batches take windows in turns of two buffers, so that a warp goes on to the next window's schedule
  // while others still fire (77 -> 75 us per epoch at 64 instances; a plain 70k-point fit 28.8 -> 29.9).
  constexpr int TURNS = SEG ? 2 : 1;
  __shared__ uint32_t s_masks[TURNS][POOL_BT];
  __shared__ uint8_t s_orders[TURNS][POOL_BT];
  __shared__ uint64_t s_base[SL];
  __shared__ uint32_t s_width[SL], s_split[SL], s_hists[TURNS][POOL_WIN + 1], s_totals[TURNS];
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint64_t slice0 = (uint64_t)blockIdx.x * SL;
  if (early) umma::grid_release();
  if (tid < SL) {
    const bool in = slice0 + tid < n_slices;
    s_base[tid] = in ? slice_base[slice0 + tid] : 0;
    s_width[tid] = in ? slice_width[slice0 + tid] : 0;
    s_split[tid] = in ? split_mask[slice0 + tid] : 0;
  }
  __syncthreads();
  uint32_t width = 0;  // the block's longest task
#pragma unroll
  for (int w = 0; w < SL; ++w) width = max(width, s_width[w]);
  for (uint32_t ew = 0; ew < width; ew += POOL_WIN) {
    const uint32_t turn = SEG ? (ew / POOL_WIN) & 1 : 0;
    uint32_t *s_mask = s_masks[turn], *s_hist = s_hists[turn], &s_total = s_totals[turn];
    uint8_t* s_order = s_orders[turn];
    if (tid <= POOL_WIN) s_hist[tid] = 0;
    {
      const uint32_t sub = lane >> 3, el = lane & 7, wd = s_width[warp];
      const uint32_t lim = ew < wd ? min(wd - ew, (uint32_t)POOL_WIN) : 0u;
      const uint2* src = entry + s_base[warp] + ew + el;
#pragma unroll 1
      for (uint32_t t = 0; t < 32; t += 16) {
        uint32_t m[4] = {0, 0, 0, 0};
#pragma unroll
        for (uint32_t h = 0; h < POOL_WIN; h += 16) {
          if (h >= lim) break;  // the same for the whole warp
          uint32_t q[8];        // 8 loads in flight before the first vote
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const uint32_t j = h + (i & 1) * 8, tt = t + (i >> 1) * 4 + sub;
            q[i] = j + el < lim ? __ldg(&src[(uint64_t)tt * wd + j].y) : 0u;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const unsigned b = __ballot_sync(0xFFFFFFFFu, fires_at(epoch, q[i]));
            m[i >> 1] |= ((b >> (8 * sub)) & 0xFFu) << (h + (i & 1) * 8);
          }
        }
        if (el == 0) {
#pragma unroll
          for (int i = 0; i < 4; ++i) s_mask[warp * 32 + t + i * 4 + sub] = m[i];
        }
      }
    }
    __syncthreads();
    const uint32_t c = __popc(s_mask[tid]);
    const unsigned peers = __match_any_sync(0xFFFFFFFFu, c);
    const int leader = __ffs(peers) - 1;
    if ((int)lane == leader) atomicAdd(&s_hist[c], (uint32_t)__popc(peers));
    __syncthreads();
    if (warp == 0) {  // s_hist[k] = number of tasks with more than k firings (k >= 1)
      const uint32_t k = 32 - lane, h = s_hist[k];
      uint32_t v = h;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, v, o);
        if ((int)lane >= o) v += u;
      }
      s_hist[k] = v - h;
      if (lane == 31) s_total = v;
    }
    __syncthreads();
    uint32_t pos = 0;
    if ((int)lane == leader && c) pos = atomicAdd(&s_hist[c], (uint32_t)__popc(peers));
    pos = __shfl_sync(0xFFFFFFFFu, pos, leader) + __popc(peers & ((1u << lane) - 1u));
    if (c) s_order[pos] = (uint8_t)tid;
    if (ew == 0) umma::grid_wait();
    __syncthreads();
    if (tid < s_total) {
      const uint32_t o = s_order[tid], sl = o >> 5, tl = o & 31;
      const uint32_t row = rowid[(slice0 + sl) * 32 + tl];
      const uint64_t first = s_base[sl] + (uint64_t)tl * s_width[sl] + ew;
      const uint2* lent = entry + first;
      uint32_t m = s_mask[o], e = (uint32_t)__ffs(m) - 1;
      uint32_t seg_lo = 0, seg_n = p.n_vertices;
      if constexpr (SEG) {
        const uint32_t sg = p.row_seg[row];
        seg_lo = (uint32_t)p.seg_off[sg];
        seg_n = (uint32_t)(p.seg_off[sg + 1] - p.seg_off[sg]);
      }
      uint2 nx = __ldg(lent + e);
      float cur[DIM], start[DIM];
      float* hrow = live + (uint64_t)row * DIM;
      load_row<DIM>(cur, hrow);
#pragma unroll
      for (int d = 0; d < DIM; ++d) start[d] = cur[d];
      if constexpr (GEN) {
        while (m) {
          const uint2 en = nx;
          const uint64_t idx = first + e;
          m &= m - 1;
          if (m) {
            e = (uint32_t)__ffs(m) - 1;
            nx = __ldg(lent + e);
          }
          fired_edge<DIM, GEN, NB_POOL, false>(cur, row, en.x, negatives_at(epoch, en.y, p.neg_rate), snap, p, alpha, idx,
                                        epoch, seg_lo, seg_n);
        }
      } else {
        // A firing's row loads are issued, then the next one's rows are drawn while they are in flight.
        constexpr bool FAR = DIM <= 2;  // the entry after that is loaded then too (wider rows would spill)
        uint32_t kk[NB_POOL], nneg, tail;
        uint64_t idx;
        auto draw = [&]() {  // rows of the firing of entry nx (the head itself: no row)
          idx = first + e;
          tail = nx.x;
          nneg = negatives_at(epoch, nx.y, p.neg_rate);
          const NegRng rng(p.seed, idx, epoch);
          uint64_t rnd = 0;
#pragma unroll
          for (int q = 0; q < NB_POOL; ++q) {
            if ((q & 1) == 0 && (q < 6 || (uint32_t)q < nneg)) rnd = rng.pair(q >> 1);
            kk[q] = (uint32_t)q < nneg ? seg_lo + __umulhi((q & 1) ? (uint32_t)(rnd >> 32) : (uint32_t)rnd, seg_n) : row;
          }
        };
        auto step = [&]() {
          m &= m - 1;
          if (m) {
            e = (uint32_t)__ffs(m) - 1;
            nx = __ldg(lent + e);
          }
        };
        auto next = [&]() {
          draw();
          if constexpr (FAR) step();
        };
        next();
        for (bool more = true; more;) {
          float o[DIM], ob[NB_POOL][DIM], g[DIM];
          float* oth = snap + (uint64_t)tail * DIM;
          load_row<DIM>(o, oth);
          uint32_t ok = 0;
#pragma unroll
          for (int q = 0; q < NB_POOL; ++q)
            if (kk[q] != row) {
              ok |= 1u << q;
              // uniform rows, rarely reused by this SM: cached in L2 only (see fired_edge); those of a
              // small instance of a batch are (64 instances, 432k points: 83 -> 77 us per epoch)
              if constexpr (DIM == 2 && !SEG) load_row_l2<DIM>(ob[q], snap + (uint64_t)kk[q] * DIM);
              else load_row<DIM>(ob[q], snap + (uint64_t)kk[q] * DIM);
            }
          const uint32_t drawn = nneg;
          const uint64_t at = idx;
          if constexpr (!FAR) step();
          more = m != 0;
          // (MANY: a firing of more negatives than fetched together still needs the arrays)
          if (more && (!MANY || drawn <= NB_POOL)) next();
          attract<DIM>(cur, o, g, p, alpha);
#pragma unroll
          for (int d = 0; d < DIM; ++d) cur[d] += g[d];
          sub_row<DIM>(oth, g);
#pragma unroll
          for (int q = 0; q < NB_POOL; ++q)
            if ((ok >> q) & 1u) repel<DIM>(cur, ob[q], p, rep, alpha);
          const NegRng rng(p.seed, at, epoch);
          if constexpr (MANY) {
            if (drawn > NB_POOL) {
              for (uint32_t q0 = NB_POOL; q0 < drawn; q0 += NB_POOL) {
                uint64_t rnd = 0;
#pragma unroll
                for (int q = 0; q < NB_POOL; ++q) {
                  if ((q & 1) == 0) rnd = rng.pair((q0 + q) >> 1);
                  kk[q] = q0 + q < drawn ? seg_lo + __umulhi((q & 1) ? (uint32_t)(rnd >> 32) : (uint32_t)rnd, seg_n) : row;
                  if (kk[q] != row) load_row_l2<DIM>(ob[q], snap + (uint64_t)kk[q] * DIM);
                }
#pragma unroll
                for (int q = 0; q < NB_POOL; ++q)
                  if (kk[q] != row) repel<DIM>(cur, ob[q], p, rep, alpha);
              }
              if (more) next();
            }
          } else {
            for (uint32_t q = NB_POOL; q < drawn; ++q) {  // rare: the rate is below NB_POOL
              const uint64_t rnd = rng.pair(q >> 1);
              const uint32_t k = seg_lo + __umulhi((q & 1) ? (uint32_t)(rnd >> 32) : (uint32_t)rnd, seg_n);
              if (k == row) continue;
              load_row_l2<DIM>(o, snap + (uint64_t)k * DIM);
              repel<DIM>(cur, o, p, rep, alpha);
            }
          }
        }
      }
      if ((s_split[sl] >> tl) & 1u) {
#pragma unroll
        for (int d = 0; d < DIM; ++d) atomicAdd(hrow + d, cur[d] - start[d]);
      } else {
        store_row<DIM>(hrow, cur);
      }
    }
    if (!SEG) __syncthreads();
  }
  if (!early) umma::grid_release();
}

// 8 columns or more (and 5 or more with the generic-metric rule): same algorithm, a thread per task,
// head row in global memory (owned by this
// lane for whole-row tasks; split tasks accumulate their delta in place with atomics).  GEN
// selects the generic-metric rule as in fired_edge.
template <bool GEN>
__global__ void __launch_bounds__(256) sgd_epoch_anydim(
    const uint64_t* __restrict__ slice_base, const uint32_t* __restrict__ slice_width,
    const uint32_t* __restrict__ split_mask, const uint32_t* __restrict__ rowid,
    const uint2* __restrict__ entry, uint64_t n_slices, float* __restrict__ live, float* snap,
    SgdParams p, uint32_t epoch, float alpha, bool lane_major) {
  const uint64_t slice = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  if (slice >= n_slices) return;
  const uint32_t r = rowid[slice * 32 + lane];
  if (r == PAD_ROW) return;
  const uint32_t width = slice_width[slice];
  const uint64_t base = slice_base[slice];
  const bool split = (split_mask[slice] >> lane) & 1u;
  uint32_t seg_lo = 0, seg_n = p.n_vertices;
  if (p.row_seg) {
    const uint32_t sg = p.row_seg[r];
    seg_lo = (uint32_t)p.seg_off[sg];
    seg_n = (uint32_t)(p.seg_off[sg + 1] - p.seg_off[sg]);
  }
  const uint32_t dim = p.dim;
  float* cur = live + (uint64_t)r * dim;
  const uint32_t n = epoch;
  const uint64_t seed = p.seed;
  const float a = p.a, b = p.b;
  auto add = [&](uint32_t d, float v) {
    if (split) atomicAdd(cur + d, v);
    else cur[d] += v;
  };
  for (uint32_t e = 0; e < width; ++e) {
    const uint64_t idx = lane_major ? base + (uint64_t)lane * width + e : base + (uint64_t)e * 32 + lane;
    const uint2 en = __ldcs(entry + idx);
    if (!fires_at(n, en.y)) continue;
    float* oth = snap + (uint64_t)en.x * dim;
    float ds = 0.0f;
    for (uint32_t d = 0; d < dim; ++d) { const float df = cur[d] - oth[d]; ds += df * df; }
    float gc = 0.0f, den = 1.0f;
    if constexpr (GEN) {
      gc = metric_coeff(ds, a, p.two_b, p.two_b, -1.0f, &den);
    } else if (ds > 0.0f) {
      const float pb = __powf(ds, b);
      gc = __fdividef(p.neg_attr * pb, ds * (a * pb * ds + 1.0f));
    }
    for (uint32_t d = 0; d < dim; ++d) {
      const float cd = cur[d], od = oth[d];
      const float g = clip4(gc * (GEN ? __fdividef(cd - od, den) : cd - od)) * alpha;
      add(d, g);
      atomicAdd(oth + d, -g);
    }
    const uint32_t nneg = negatives_at(n, en.y, p.neg_rate);
    const NegRng rng(seed, idx, epoch);
    uint64_t rnd = 0;
    for (uint32_t q = 0; q < nneg; ++q) {
      if ((q & 1) == 0) rnd = rng.pair(q >> 1);
      const uint32_t rv = (q & 1) ? (uint32_t)(rnd >> 32) : (uint32_t)rnd;
      const uint32_t kk = seg_lo + __umulhi(rv, seg_n);
      if (kk == r) continue;
      const float* ob = snap + (uint64_t)kk * dim;
      float dsn = 0.0f;
      for (uint32_t d = 0; d < dim; ++d) { const float df = cur[d] - ob[d]; dsn += df * df; }
      if constexpr (GEN) {
        float dn;
        const float gr = metric_coeff(dsn, a, p.two_b, p.pos_rep, 0.0f, &dn);
        for (uint32_t d = 0; d < dim; ++d) add(d, clip4(gr * __fdividef(cur[d] - ob[d], dn)) * alpha);
      } else {
        float gr = 0.0f;
        if (dsn > 0.0f) {
          const float pb = __powf(dsn, b);
          gr = __fdividef(p.pos_rep, (0.001f + dsn) * (a * pb * dsn + 1.0f));
        }
        if (gr > 0.0f)
          for (uint32_t d = 0; d < dim; ++d) add(d, clip4(gr * (cur[d] - ob[d])) * alpha);
      }
    }
  }
}

// Rows of 5 to 7 columns: a thread per task with its head row in registers, a firing's tail and
// negative rows fetched together, the warp's lanes at the same entry.  A task that is a part of a
// row adds each move to the live row and reads it back, so that the parts of a row move together;
// one merge per firing runs twice as fast (48 us), but by then the layouts differ from one another
// by up to eight times as much as two runs do.  sgd_epoch_anydim, which keeps the head row in global memory, pays a
// dependent round trip per column instead (20k points, 5-D: 515 us per epoch, here 106; 3,000: 396,
// here 93).  What is left is the chain of read-backs of the partial rows.
template <int DIM>
__global__ void __launch_bounds__(256) sgd_epoch_rows(
    const uint64_t* __restrict__ slice_base, const uint32_t* __restrict__ slice_width,
    const uint32_t* __restrict__ split_mask, const uint32_t* __restrict__ rowid,
    const uint2* __restrict__ entry, uint64_t n_slices, float* __restrict__ live, float* snap,
    SgdParams p, uint32_t epoch, float alpha) {
  constexpr int NB = 6;  // negative rows fetched together
  const float rep = fmaxf(p.pos_rep, 0.0f);
  const uint64_t slice = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t lane = threadIdx.x & 31;
  if (slice >= n_slices) return;
  const uint32_t r = rowid[slice * 32 + lane];
  if (r == PAD_ROW) return;
  const uint32_t width = slice_width[slice];
  const uint64_t first = slice_base[slice] + (uint64_t)lane * width;
  const bool split = (split_mask[slice] >> lane) & 1u;
  uint32_t seg_lo = 0, seg_n = p.n_vertices;
  if (p.row_seg) {
    const uint32_t sg = p.row_seg[r];
    seg_lo = (uint32_t)p.seg_off[sg];
    seg_n = (uint32_t)(p.seg_off[sg + 1] - p.seg_off[sg]);
  }
  float* hrow = live + (uint64_t)r * DIM;
  float cur[DIM];
  load_row<DIM>(cur, hrow);
  auto move = [&](const float (&g)[DIM]) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
      cur[d] += g[d];
      if (split) atomicAdd(hrow + d, g[d]);
    }
  };
  for (uint32_t ew = 0; ew < width; ew += 4) {  // width is a multiple of 4 (slice_meta_kernel)
    uint2 win[4];
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(entry + first + ew + j));
      win[j] = make_uint2(v.x, v.y);
      win[j + 1] = make_uint2(v.z, v.w);
    }
#pragma unroll 1
    for (uint32_t j = 0; j < 4; ++j) {
      const uint2 en = j == 0 ? win[0] : j == 1 ? win[1] : j == 2 ? win[2] : win[3];
      if (!fires_at(epoch, en.y)) continue;
      float* oth = snap + (uint64_t)en.x * DIM;
      const uint32_t nneg = negatives_at(epoch, en.y, p.neg_rate);
      const NegRng rng(p.seed, first + ew + j, epoch);
      float o[DIM], g[DIM], df[DIM], x[NB][DIM];
      uint32_t kk[NB];
      if (split) load_row_l2<DIM>(cur, hrow);
      load_row<DIM>(o, oth);
      auto fetch = [&](uint32_t q0) {  // negatives q0 .. q0 + NB - 1 (the head itself: none)
        uint64_t rnd = 0;
#pragma unroll
        for (int q = 0; q < NB; ++q) {
          if ((q & 1) == 0) rnd = rng.pair((q0 + q) >> 1);
          kk[q] = q0 + q < nneg ? seg_lo + __umulhi((q & 1) ? (uint32_t)(rnd >> 32) : (uint32_t)rnd, seg_n) : r;
          if (kk[q] != r) load_row<DIM>(x[q], snap + (uint64_t)kk[q] * DIM);
        }
      };
      fetch(0);
      // attractive step (optimize_layout_euclidean.rs:284-306)
      {
        attract<DIM>(cur, o, g, p, alpha);
        move(g);
        sub_row<DIM>(oth, g);
      }
      // negative samples (:313-341)
      for (uint32_t q0 = 0; q0 < nneg; q0 += NB) {
        if (q0 > 0) fetch(q0);
#pragma unroll
        for (int q = 0; q < NB; ++q) {
          if (kk[q] == r) continue;
          if (split) load_row_l2<DIM>(cur, hrow);
#pragma unroll
          for (int d = 0; d < DIM; ++d) df[d] = cur[d] - x[q][d];
          if (!repel_move<DIM>(df, g, p, rep)) continue;
#pragma unroll
          for (int d = 0; d < DIM; ++d) g[d] *= alpha;
          move(g);
        }
      }
    }
  }
  if (!split) store_row<DIM>(hrow, cur);
}

// ------------------------------------------------------------------------------ K5 pieces
__global__ void kept_degree_kernel(const uint64_t* __restrict__ indptr, const float* __restrict__ data,
                                   uint64_t n, float thr, const float* __restrict__ seg_thr,
                                   const uint32_t* __restrict__ row_seg, uint32_t* __restrict__ deg) {
  const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const float t = seg_thr ? seg_thr[row_seg[r]] : thr;
  uint32_t c = 0;
  for (uint64_t q = indptr[r]; q < indptr[r + 1]; ++q) c += data[q] >= t ? 1u : 0u;
  deg[r] = c;
}

// Batched instances: max graph weight of each instance (optimizer.rs:90-94 per instance).  gridDim.y
// blocks share an instance and merge by its bits (the maximum is at least +0): 64 instances of 75k
// edges took 357 us with a block each, 25 with 18.
__global__ void segment_max_kernel(const uint64_t* __restrict__ indptr, const float* __restrict__ data,
                                   const uint64_t* __restrict__ seg_off, int* __restrict__ out) {
  const uint32_t sgm = blockIdx.x;
  const uint64_t q0 = indptr[seg_off[sgm]], q1 = indptr[seg_off[sgm + 1]];
  float m = 0.0f;
  const uint64_t step = (uint64_t)gridDim.y * blockDim.x;
#pragma unroll 4
  for (uint64_t q = q0 + blockIdx.y * blockDim.x + threadIdx.x; q < q1; q += step) m = fmaxf(m, data[q]);
  __shared__ float s_m[32];
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t w = 1; w < blockDim.x / 32; ++w) m = fmaxf(m, s_m[w]);
    atomicMax(out + sgm, __float_as_int(m));
  }
}

// Row u of the layout is row order[u] of the kept-edge CSR (order null: the same row).
__global__ void ptr_degree_kernel(const uint64_t* __restrict__ kptr, uint64_t n, uint32_t chunk,
                                  const uint32_t* __restrict__ order, uint32_t* __restrict__ deg,
                                  uint32_t* __restrict__ ntask) {
  const uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= n) return;
  const uint64_t r = order ? order[u] : u;
  const uint32_t d = (uint32_t)(kptr[r + 1] - kptr[r]);
  deg[u] = d;
  ntask[u] = (d + chunk - 1) / chunk;
}

// One task per chunk of a row: row id, first kept-edge index, length, split flag, sort key.
// The key orders tasks by descending length and, with rate_bits = RATE_BITS, then by
// descending mean firing rate (sum over the task's edges of min(1, 1 / epochs_per_sample),
// over its length, in RATE_BITS bits), so that a warp's lanes draw similar numbers of firings
// per epoch; batched instances sort instance-major first.
constexpr int RATE_BITS = 8;
// With rates, G = 16 lanes per row: the divisions of 16 edges at once, added up in their order (10k
// points: 63 us with a thread per row, 18 with 16); without, G = 1.
template <int G>
__global__ void task_fill_kernel(const uint64_t* __restrict__ kptr, const uint32_t* __restrict__ deg,
                                 const uint64_t* __restrict__ tptr, uint64_t n, uint32_t chunk,
                                 const uint32_t* __restrict__ row_seg, int len_bits, int rate_bits,
                                 int block_shift, const double* __restrict__ keps, const uint32_t* __restrict__ order,
                                 uint32_t* __restrict__ trow, uint64_t* __restrict__ tstart,
                                 uint32_t* __restrict__ tkey) {
  const uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
  if (r >= n) return;
  const uint32_t gl = threadIdx.x & (G - 1), gmask = ((1u << G) - 1u) << (threadIdx.x & 31 & ~(G - 1));
  const uint64_t src = order ? order[r] : r;  // the kept-edge CSR row of layout row r
  const uint32_t d = deg[r];
  const uint64_t t0 = tptr[r], nt = tptr[r + 1] - t0;
  for (uint64_t c = 0; c < nt; ++c) {
    const uint32_t len = (uint32_t)min((uint64_t)chunk, (uint64_t)d - c * chunk);
    const uint64_t st = kptr[src] + c * chunk;
    uint32_t rate = 0;
    if (rate_bits) {
      float sp = 0.0f;
      for (uint32_t e = 0; e < len; e += G) {
        const double x = e + gl < len ? keps[st + e + gl] : 0.0;
        const float p = x > 1.0 ? (float)(1.0 / x) : (x > 0.0 ? 1.0f : 0.0f);
#pragma unroll
        for (int i = 0; i < G; ++i) sp += __shfl_sync(gmask, p, i, G);  // past the end: + 0
      }
      const uint32_t top = (1u << rate_bits) - 1u;
      rate = top - min(top, (uint32_t)(sp / (float)max(len, 1u) * (float)(top + 1u)));
    }
    const uint32_t hi = block_shift >= 0 ? (uint32_t)(r >> block_shift) : (row_seg ? row_seg[r] : 0u);
    if (gl == 0) {
      trow[t0 + c] = (uint32_t)r | (nt > 1 ? 0x80000000u : 0u);   // high bit: partial row
      tstart[t0 + c] = st;
      tkey[t0 + c] = (((hi << len_bits) | (chunk - len)) << rate_bits) | rate;
    }
  }
}

__global__ void iota_u32_kernel(uint32_t* __restrict__ p, uint64_t n) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = (uint32_t)i;
}

__global__ void slice_meta_kernel(const uint32_t* __restrict__ perm, const uint32_t* __restrict__ trow,
                                  const uint32_t* __restrict__ skey, uint64_t T, uint64_t n_slices,
                                  uint32_t chunk, int rate_bits, uint32_t len_mask, bool lane_major,
                                  uint32_t* __restrict__ width,
                                  uint32_t* __restrict__ rowid, uint32_t* __restrict__ split_mask) {
  const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n_slices * 32) return;
  const uint32_t tr = q < T ? trow[perm[q]] : PAD_ROW;
  rowid[q] = tr == PAD_ROW ? PAD_ROW : (tr & 0x7FFFFFFFu);
  const unsigned bits = __ballot_sync(0xFFFFFFFFu, tr != PAD_ROW && (tr & 0x80000000u));
  // slice width = longest task of the slice (instance-major order: the max over lanes)
  uint32_t len = q < T ? chunk - ((skey[q] >> rate_bits) & len_mask) : 0u;
  for (int o = 16; o > 0; o >>= 1) len = max(len, __shfl_xor_sync(0xFFFFFFFFu, len, o));
  // whole 32-byte sectors per task
  if (lane_major) len = (len + 3u) / 4u * 4u;
  if ((q & 31) == 0) {
    width[q >> 5] = len;
    split_mask[q >> 5] = bits;
  }
}

// The entries of the tasks: 8 lanes per task where a task's entries are contiguous, a lane per task where
// they are interleaved, so that a warp's writes fill whole sectors in both (2M points, lane major: 708
// us with a lane per task, 327 with 8).
__global__ void slice_fill_kernel(const uint32_t* __restrict__ ktail, const double* __restrict__ keps,
                                  const uint32_t* __restrict__ perm, const uint64_t* __restrict__ tstart,
                                  const uint32_t* __restrict__ skey, uint64_t T, uint32_t chunk,
                                  int rate_bits, uint32_t len_mask, const uint64_t* __restrict__ wscan,
                                  const uint32_t* __restrict__ width, uint64_t n_slices, bool lane_major,
                                  const uint32_t* __restrict__ rank, uint2* __restrict__ entry) {
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, q = lane_major ? t >> 3 : t;
  if (q >= n_slices * 32) return;
  const uint64_t s = q >> 5;
  const uint32_t lane = (uint32_t)(q & 31), wd = width[s], step = lane_major ? 8 : 1;
  const uint64_t base = wscan[s] * 32 + (lane_major ? (uint64_t)lane * wd : lane), stride = lane_major ? 1 : 32;
  const uint64_t st = q < T ? tstart[perm[q]] : 0;
  const uint32_t len = q < T ? chunk - ((skey[q] >> rate_bits) & len_mask) : 0u;
  for (uint32_t e = lane_major ? (uint32_t)t & 7 : 0u; e < wd; e += step) {
    uint2 v = make_uint2(0u, 0u);
    if (e < len) v = make_uint2(rank ? rank[ktail[st + e]] : ktail[st + e], q_minus_1(keps[st + e]));
    entry[base + e * stride] = v;
  }
}

__global__ void head_from_ptr_kernel(const uint64_t* __restrict__ kptr, uint64_t n, uint32_t* __restrict__ head) {
  const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  for (uint64_t j = kptr[r]; j < kptr[r + 1]; ++j) head[j] = (uint32_t)r;
}

// Schedule state of the reference at `cur` (optimizer.rs:41-43) from the closed form:
// m = firings so far, T = negatives drawn so far;  eons = (m+1)*eps, epns = eps/neg,
// eonns = epns*(1+T).
__global__ void export_state_kernel(const double* __restrict__ eps, uint64_t E, uint64_t neg,
                                    uint64_t cur, double* __restrict__ eons, double* __restrict__ eonns,
                                    double* __restrict__ epns) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= E) return;
  const double e = eps[i];
  const uint32_t q = q_minus_1(e);
  const uint64_t m = cur > 0 ? fires_by((uint32_t)(cur - 1), q) : 0ull;
  const uint64_t t = negatives_after(m, q, (uint32_t)neg);
  const double pn = e / (double)neg;
  if (eons) eons[i] = e * ((double)m + 1.0);
  if (epns) epns[i] = pn;
  if (eonns) eonns[i] = pn * (1.0 + (double)t);
}

// make_epochs_per_sample.rs:30-49 in f64.
__device__ __forceinline__ double epochs_per_sample(float w, double max_w, double n_ep) {
  const double n_samples = n_ep * ((double)w / max_w);
  return n_samples > 0.0 ? n_ep / n_samples : -1.0;
}

// 8 lanes per row, their kept edges placed by rank, so that reads and writes fill sectors (2M points: 1117
// us with a thread per row, 696 with 8 lanes).
__global__ void export_edges_kernel(const uint64_t* __restrict__ indptr, const uint32_t* __restrict__ indices,
                                    const float* __restrict__ data, uint64_t n, float thr, double max_w,
                                    double n_ep, const float* __restrict__ seg_thr,
                                    const float* __restrict__ seg_maxw, const uint32_t* __restrict__ row_seg,
                                    const uint64_t* __restrict__ kept_ptr, uint32_t* __restrict__ head,
                                    uint32_t* __restrict__ tail, double* __restrict__ eps) {
  constexpr uint32_t G = 8;
  const uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
  if (r >= n) return;
  const uint32_t gl = threadIdx.x & (G - 1), shift = threadIdx.x & 24, gmask = 0xFFu << shift;
  float t = thr;
  double mw = max_w;
  if (seg_thr) {
    const uint32_t sg = row_seg[r];
    t = seg_thr[sg];
    mw = (double)seg_maxw[sg];
  }
  uint64_t o = kept_ptr[r];
  const uint64_t jend = indptr[r + 1];
  for (uint64_t jb = indptr[r]; jb < jend; jb += G) {
    const uint64_t j = jb + gl;
    const float w = j < jend ? data[j] : 0.0f;
    const uint32_t k = tail && j < jend ? indices[j] : 0;
    const bool keep = j < jend && w >= t;
    const uint32_t bits = (__ballot_sync(gmask, keep) & gmask) >> shift;
    if (keep) {
      const uint64_t at = o + __popc(bits & ((1u << gl) - 1u));
      if (head) head[at] = (uint32_t)r;
      if (tail) tail[at] = k;
      if (eps) eps[at] = epochs_per_sample(w, mw, n_ep);
    }
    o += __popc(bits);
  }
}

// ------------------------------------------------------------------------------ K6
// optimizer.rs:189-230.  f32::min / f32::max ignore NaN like fminf / fmaxf.
__global__ void minmax_dim_kernel(const float* __restrict__ emb, uint64_t n, uint32_t dim,
                                  const uint64_t* __restrict__ seg_off, float* __restrict__ mins,
                                  float* __restrict__ scales) {
  // one block per (dimension, instance)
  const uint32_t d = blockIdx.x, sg = blockIdx.y;
  const uint64_t r0 = seg_off ? seg_off[sg] : 0, r1 = seg_off ? seg_off[sg + 1] : n;
  float mn = INFINITY, mx = -INFINITY;
  for (uint64_t i = r0 + threadIdx.x; i < r1; i += blockDim.x) {
    const float v = emb[i * dim + d];
    mn = fminf(mn, v);
    mx = fmaxf(mx, v);
  }
  __shared__ float s_mn[32], s_mx[32];
  for (int o = 16; o > 0; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xFFFFFFFFu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
  }
  if ((threadIdx.x & 31) == 0) { s_mn[threadIdx.x >> 5] = mn; s_mx[threadIdx.x >> 5] = mx; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t w = 1; w < blockDim.x / 32; ++w) { mn = fminf(mn, s_mn[w]); mx = fmaxf(mx, s_mx[w]); }
    const float range = __fsub_rn(mx, mn);
    mins[sg * dim + d] = mn;
    scales[sg * dim + d] = range > 0.0f ? __fdiv_rn(10.0f, range) : 0.0f;
  }
}

// A plain fit's column min / max in two stages: block b of dimension d reduces rows
// b, b + G, ... into part[d][b]; then minmax_finish_kernel folds the G partials.  Min and max
// ignore NaN and are exact in any order, so the result equals one block's.
__global__ void minmax_part_kernel(const float* __restrict__ emb, uint64_t n, uint32_t dim,
                                   float* __restrict__ pmin, float* __restrict__ pmax) {
  const uint32_t d = blockIdx.y, G = gridDim.x;
  float mn = INFINITY, mx = -INFINITY;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)G * blockDim.x) {
    const float v = emb[i * dim + d];
    mn = fminf(mn, v);
    mx = fmaxf(mx, v);
  }
  __shared__ float s_mn[32], s_mx[32];
  for (int o = 16; o > 0; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xFFFFFFFFu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
  }
  if ((threadIdx.x & 31) == 0) { s_mn[threadIdx.x >> 5] = mn; s_mx[threadIdx.x >> 5] = mx; }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (uint32_t w = 1; w < blockDim.x / 32; ++w) { mn = fminf(mn, s_mn[w]); mx = fmaxf(mx, s_mx[w]); }
    pmin[d * G + blockIdx.x] = mn;
    pmax[d * G + blockIdx.x] = mx;
  }
}

__global__ void minmax_finish_kernel(const float* __restrict__ pmin, const float* __restrict__ pmax, uint32_t G,
                                     float* __restrict__ mins, float* __restrict__ scales) {
  const uint32_t d = blockIdx.x;
  float mn = INFINITY, mx = -INFINITY;
  for (uint32_t g = threadIdx.x; g < G; g += blockDim.x) {
    mn = fminf(mn, pmin[d * G + g]);
    mx = fmaxf(mx, pmax[d * G + g]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xFFFFFFFFu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
  }
  if (threadIdx.x == 0) {
    const float range = __fsub_rn(mx, mn);
    mins[d] = mn;
    scales[d] = range > 0.0f ? __fdiv_rn(10.0f, range) : 0.0f;
  }
}

__global__ void normalize_kernel(float* __restrict__ emb, uint64_t total, uint32_t dim,
                                 const float* __restrict__ mins, const float* __restrict__ scales,
                                 const uint32_t* __restrict__ row_seg) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  const uint64_t r = i / dim;
  const uint32_t d = (uint32_t)(i - r * dim);
  const uint64_t c = (uint64_t)(row_seg ? row_seg[r] : 0) * dim + d;
  const float sc = scales[c];
  if (sc > 0.0f) emb[i] = __fmul_rn(__fsub_rn(emb[i], mins[c]), sc);
}

// ------------------------------------------------------------------------------ accounting
__global__ void schedule_totals_kernel(const uint2* __restrict__ entry, uint64_t n_entries, uint64_t neg,
                                       uint64_t start, uint64_t end, unsigned long long* __restrict__ fired,
                                       unsigned long long* __restrict__ negs) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long f = 0, g = 0;
  if (i < n_entries) {
    const uint32_t q = entry[i].y;
    // firings in [start, end) = m(end-1) - m(start-1); negatives telescope the same way.
    const uint64_t fe = end > 0 ? fires_by((uint32_t)(end - 1), q) : 0ull;
    const uint64_t fs = start > 0 ? fires_by((uint32_t)(start - 1), q) : 0ull;
    f = fe - fs;
    g = negatives_after(fe, q, (uint32_t)neg) - negatives_after(fs, q, (uint32_t)neg);
  }
  for (int o = 16; o > 0; o >>= 1) {
    f += __shfl_xor_sync(0xFFFFFFFFu, f, o);
    g += __shfl_xor_sync(0xFFFFFFFFu, g, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (f) atomicAdd(fired, f);
    if (g) atomicAdd(negs, g);
  }
}

// The negative samples the epoch kernel would draw for the firings of entries
// [first, first + count) at `epoch`: draw q of entry e is out[(e - first) * per + q], made by
// the same generator and mapping as fired_edge (half q & 1 of pair q >> 1, multiply-high into
// [lo, lo + range)).  Statistical tests of the generator read these.
__global__ void negative_draws_kernel(uint64_t seed, uint64_t first, uint64_t count, uint32_t epoch,
                                      uint32_t per, uint32_t lo, uint32_t range, uint32_t* __restrict__ out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const NegRng rng(seed, first + i, epoch);
  uint64_t rnd = 0;
  for (uint32_t q = 0; q < per; ++q) {
    if ((q & 1) == 0) rnd = rng.pair(q >> 1);
    const uint32_t rv = (q & 1) ? (uint32_t)(rnd >> 32) : (uint32_t)rnd;
    out[i * per + q] = lo + __umulhi(rv, range);
  }
}

// Negatives the epoch kernel draws for a firing of an entry with schedule word q at epoch n
// (0 where the entry does not fire at n): the schedule's per-firing count, for exact tests.
__global__ void negatives_per_firing_kernel(const uint32_t* __restrict__ qs, const uint32_t* __restrict__ ns,
                                            uint64_t count, uint32_t neg, uint32_t* __restrict__ out) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const uint32_t q = qs[i], n = ns[i];
  out[i] = fires_at(n, q) ? negatives_at(n, q, neg) : 0u;
}

__global__ void nan_rows_kernel(const uint64_t* __restrict__ indptr, uint64_t n, uint32_t dim,
                                float* __restrict__ emb) {
  const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n || indptr[r + 1] != indptr[r]) return;
  for (uint32_t d = 0; d < dim; ++d) emb[r * dim + d] = __int_as_float(0x7FC00000);
}

__global__ void scale32_kernel(uint64_t* __restrict__ x, uint64_t n) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i] *= 32;
}

inline unsigned grid_for(uint64_t n, unsigned bt) { return (unsigned)((n + bt - 1) / bt); }

}  // namespace

void kept_degree(const uint64_t* indptr, const float* data, uint64_t n, float thr, uint32_t* deg,
                 cudaStream_t s, const SegmentPrune* sp) {
  if (n == 0) return;
  kept_degree_kernel<<<grid_for(n, 256), 256, 0, s>>>(indptr, data, n, thr, sp ? sp->seg_thr : nullptr,
                                                      sp ? sp->row_seg : nullptr, deg);
  UB_LAUNCH_CHECK();
}

void segment_max(const uint64_t* indptr, const float* data, const uint64_t* seg_off, uint32_t n_seg,
                 float* out, cudaStream_t s) {
  if (n_seg == 0) return;
  UB_CUDA(cudaMemsetAsync(out, 0, n_seg * sizeof(float), s));
  const unsigned parts = std::max(1u, std::min(64u, 1184u / n_seg));  // about 8 blocks per SM in all
  segment_max_kernel<<<dim3(n_seg, parts), 256, 0, s>>>(indptr, data, seg_off, (int*)out);
  UB_LAUNCH_CHECK();
}

void prune_edges(const uint64_t* indptr, const float* data, uint64_t n, float thr, uint64_t* kept_ptr,
                 uint64_t* n_edges, cudaStream_t s, const SegmentPrune* sp) {
  DevBuf<uint32_t> deg(n, s);
  kept_degree(indptr, data, n, thr, deg.p, s, sp);
  scan_u32_to_u64(deg.p, kept_ptr, n, s);
  UB_CUDA(cudaMemcpyAsync(n_edges, kept_ptr + n, 8, cudaMemcpyDeviceToHost, s));
  UB_CUDA(cudaStreamSynchronize(s));
}

void head_from_ptr(const uint64_t* kept_ptr, uint64_t n, uint32_t* head, cudaStream_t s) {
  if (n == 0) return;
  head_from_ptr_kernel<<<grid_for(n, 256), 256, 0, s>>>(kept_ptr, n, head);
  UB_LAUNCH_CHECK();
}

void export_state(const double* eps, uint64_t E, uint64_t neg_rate, uint64_t cur_epoch, double* eons,
                  double* eonns, double* epns, cudaStream_t s) {
  if (E == 0) return;
  export_state_kernel<<<grid_for(E, 256), 256, 0, s>>>(eps, E, neg_rate, cur_epoch, eons, eonns, epns);
  UB_LAUNCH_CHECK();
}

// Longest task (edges) so that no single lane's chain of updates outlasts roughly half an
// epoch: an epoch streams E edges across the whole GPU, while one lane works through its
// task sequentially, so the bound grows linearly with E (~E/135k for this kernel).
uint32_t pick_chunk(uint64_t n_edges) {
  if (const char* e = getenv("UMAP_B200_CHUNK")) {
    long v = atol(e);
    if (v >= 1 && v <= (1 << 30)) return (uint32_t)v;
  }
  uint64_t c = (n_edges / 135000 + 4) / 8 * 8;
  return (uint32_t)std::min<uint64_t>(512, std::max<uint64_t>(16, c));
}

// The generic-metric rule (optimize_layout_generic.rs) attracts much harder than the
// Euclidean one, and a row cut into tasks that all start from the same head position
// overshoots where the reference applies the row's moves one after another: on the 10k-point
// Gaussian workload (4 seeds each) 16-edge tasks gave 15-NN recall 0.0348 and fuzzy
// cross-entropy 268,541 against the oracle's 0.0380 and 270,403; 32: 0.0356 / 268,666;
// 64: 0.0369 / 269,976; 128 and whole rows: no further change.  The Euclidean rule showed no
// such dependence at any task length.  So the generic rule keeps typical rows whole (tasks
// of at least 64 edges, about three times a kNN graph's mean degree) and splits only hubs.
uint32_t pick_chunk_generic(uint64_t n_edges) {
  if (getenv("UMAP_B200_CHUNK")) return pick_chunk(n_edges);
  return std::max<uint32_t>(64, pick_chunk(n_edges));
}

int sm_count() {
  int dev = 0, sms = 0;
  UB_CUDA(cudaGetDevice(&dev));
  UB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  return std::max(sms, 1);
}

// Graphs of at most two waves of a lane per task at 40 warps per SM: their tasks are ordered by firing
// rate too (pick_task_order), and the lane kernel takes its 8-negatives budget in 1-D and 2-D.
// UMAP_B200_SGD_SHORT=0 / 1 forces it, and with it the lane kernel (1-D to 4-D).
bool small_graph(uint64_t n_slices) {
  if (const char* e = getenv("UMAP_B200_SGD_SHORT")) {
    if (e[0] == '0') return false;
    if (e[0] == '1') return true;
  }
  return n_slices <= 2ull * (uint64_t)sm_count() * 40;
}

// The epoch kernel of a layout.
//  * Dram: renamed 1-D and 2-D layouts whose snapshot (4 * dim bytes per vertex) is above 80 MB, so
//    that with the edge stream it does not stay in the 126 MB L2.  The random rows then cost DRAM
//    bursts, and the interleaved order's whole 256-byte rows per warp use them better than a task's
//    contiguous entries (2-D rolls, 30 epochs, Dram interleaved against Pool lane major, ms: 5M points
//    34.7 / 28.2, 8M 55.1 / 44.6, 12M 94.6 / 98.7, 16M 149.6 / 156.9, 20M 207.2 / 221.6).
//  * Pool (1-D to 4-D) and Rows (5-D to 7-D, Euclidean rule): layouts at learning rates from which on
//    the epochs' races decide the result.  Lane and AnyDim: the others.
//    The kernels draw the same samples and make the same moves, but which updates of an epoch see
//    which differs between them, the same way in every epoch.  At small rates the races of one kernel
//    nearly average out and this difference does not: the median relative distance between runs of
//    Pool and of Lane, over that between two runs of Lane, is, at rate 0.002, 4.3 at 200k, 4.6 at 1M
//    and 2.6 at 2M points; at 0.006, 2.2 to 2.9 at 500, in 3-D 3.9 at 2,000; at 0.01, 1.7 at 300 to 1,500,
//    1.5 at 10k, 1.7 at 70k, in batches 1.6 to 2.3, in 3-D 2.0 at 10k; in 2-D at 0.05, 1.0 to 1.4; in 3-D at
//    0.1, 1.1 to 1.3, at 0.3, 1.0; Rows against AnyDim in 5-D: 4.6 at 500 and 2.8 at 100k at 0.01, 1.1 to 2.4
//    at 0.03, 1.0 at 0.3.  The lines are the rates from which on runs of the two kernels are within four
//    times the distance between two runs of one as often as those runs themselves: RACING_RATE for plain 1-D
//    and 2-D Euclidean layouts of at least POOL_MIN_SLICES slices per SM (7,500 points of 25 neighbours
//    hold it, 3,000 of 15 do not, 22% of the pairs against 3%), RACING_RATE_WIDE for the rest.
//    Renamed layouts take Pool at every rate: their locality order alone moves two runs as far apart as
//    the kernels (5M points: 7.2e-3 either way).
//    Time, Lane / Pool, ms per fit: 10k points 7.3 / 4.3, 70k 9.1 / 6.9, 1M 35.4 / 28.2, 64 instances
//    23.6 / 16.7; AnyDim / Rows, 20k points in 5-D 50 / 11.
// UMAP_B200_SGD_KERNEL=lane / pool / dram / rows / any forces one that can run the layout.
constexpr float RACING_RATE = 0.01f, RACING_RATE_WIDE = 0.03f;
constexpr double POOL_MIN_SLICES = 2.5;
constexpr uint64_t LANE_MAJOR_MAX = 4000000;
EpochKernel pick_epoch_kernel(uint64_t n, uint32_t dim, uint64_t n_slices, bool renamed, bool segmented, bool generic,
                              float alpha) {
  const char* e = getenv("UMAP_B200_SGD_KERNEL");
  const auto forced = [&](const char* name) { return e && !strcmp(e, name); };
  if (dim > 4) {
    if (dim > 7 || generic || forced("any")) return EpochKernel::AnyDim;
    return forced("rows") || alpha >= RACING_RATE_WIDE ? EpochKernel::Rows : EpochKernel::AnyDim;
  }
  const bool can_dram = dim <= 2 && !generic && !segmented;
  if (forced("dram") && can_dram) return EpochKernel::Dram;
  if (forced("pool")) return EpochKernel::Pool;
  if (forced("lane") || getenv("UMAP_B200_SGD_SHORT")) return EpochKernel::Lane;
  if (can_dram && renamed && n * dim * 4 > 80000000ull) return EpochKernel::Dram;
  if (renamed) return EpochKernel::Pool;
  if (!segmented && n > LANE_MAJOR_MAX) return EpochKernel::Lane;  // interleaved entries
  const bool early = can_dram && (double)n_slices >= POOL_MIN_SLICES * sm_count();
  return alpha >= (early ? RACING_RATE : RACING_RATE_WIDE) ? EpochKernel::Pool : EpochKernel::Lane;
}

// Entry order of the layout: lane major, or interleaved for Dram and, above 4M vertices of a plain fit,
// for the kernels that take either (their random rows go to DRAM there, whose bursts whole 256-byte rows
// per warp use better than a lane's 32-byte windows).  UMAP_B200_SGD_LANE_MAJOR=0 / 1 forces those.
bool lane_major_entries(uint64_t n, bool segmented, EpochKernel kernel) {
  if ((kernel == EpochKernel::Lane && !segmented) || kernel == EpochKernel::AnyDim) {
    if (const char* e = getenv("UMAP_B200_SGD_LANE_MAJOR")) {
      if (e[0] == '0') return false;
      if (e[0] == '1') return true;
    }
    return segmented || n <= LANE_MAJOR_MAX;
  }
  return kernel != EpochKernel::Dram;
}

// Whether a plain fit's layout renames its vertices into a locality order (order.cu): from the
// sizes at which random rows of the caller's order mostly miss L2.
// UMAP_B200_RELABEL=0 / 1 forces either.  The generic-metric rule never renames
// (build_sgd_layout): it is sensitive to which rows update at the same time (its split
// rows showed that), and its parity with the reference was established in the caller's order;
// on a 6,000-point roll one renamed run sat 2.6% from a plain one, inside that small case's
// run-to-run spread, so renaming is not shown to move it, only not shown to be harmless.
bool pick_relabel(uint64_t n, bool segmented) {
  if (segmented) return false;
  if (const char* e = getenv("UMAP_B200_RELABEL")) {
    if (e[0] == '0') return false;
    if (e[0] == '1') return true;
  }
  return n > LANE_MAJOR_MAX;
}

// Order in which the tasks are dealt to warps (32 consecutive tasks per warp):
//  * Length: descending length (a warp's lanes scan equally long tasks; least padding).
//  * LengthRate: length, then descending mean firing rate, so that a warp's lanes draw similar
//    numbers of firings per epoch.  Small graphs, whose epochs are short and bound by their
//    warps' busiest lanes (100k-point fit: 25.4-25.6 against 26.0-26.1 ms).
//  * RowBlock: blocks of 2^TASK_BLOCK_SHIFT consecutive layout rows, length order inside each.
//    Renamed layouts: their warps in flight then cover a narrow range of new ids, whose tails
//    stay in L2 (30 epochs of the 20M-point roll: 292.6 ms in length order, 245.7 in row
//    order, blocks of 2^6 / 2^8 / 2^10 / 2^12 / 2^14 / 2^16 rows: 241.4 / 237.7 / 235.6 /
//    235.3-239.1 / 239.7 / 242.9 ms; 40M points, 24 epochs: 564.7 -> 475.9 ms).
//  * Row: layout row order (measurement only; the 2M-point fit takes 5x as long in it, its
//    whole-row tasks of very different lengths padded to the longest of each warp).
// Plain fits without renaming keep Length at any size that is not short (2M points: 320.6 in
// LengthRate against 321.0 ms, within noise; a block order: 1106 ms).  Batched instances take
// LengthRate inside each instance (4,096 instances, 200 epochs: 2,822-2,825 against
// 2,842-2,843 ms per batch).  UMAP_B200_TASK_ORDER=len / rate / block / row forces one.
constexpr int TASK_BLOCK_SHIFT = 12;
TaskOrder pick_task_order(bool renamed, bool short_graph, bool segmented) {
  if (const char* e = getenv("UMAP_B200_TASK_ORDER")) {
    if (!strcmp(e, "len")) return TaskOrder::Length;
    if (!strcmp(e, "rate")) return TaskOrder::LengthRate;
    if (!strcmp(e, "block") && !segmented) return TaskOrder::RowBlock;
    if (!strcmp(e, "row")) return TaskOrder::Row;
  }
  if (segmented) return TaskOrder::LengthRate;
  if (renamed) return TaskOrder::RowBlock;
  return short_graph ? TaskOrder::LengthRate : TaskOrder::Length;
}

void build_sgd_layout(const uint64_t* kept_ptr, const uint32_t* ktail, const double* keps, uint64_t n, uint32_t dim,
                      uint32_t chunk, bool generic, float alpha, SgdLayout& L, cudaStream_t s, const Segments* seg) {
  L.n_vertices = n;
  DevBuf<uint32_t> rank;
  L.order.reset();
  if (n && !generic && pick_relabel(n, seg != nullptr)) {
    L.order.alloc(n, s);
    rank.alloc(n, s);
    locality_order(kept_ptr, ktail, n, L.order.p, rank.p, s);
  }
  uint64_t n_edges = 0;
  UB_CUDA(cudaMemcpyAsync(&n_edges, kept_ptr + n, 8, cudaMemcpyDeviceToHost, s));
  UB_CUDA(cudaStreamSynchronize(s));
  L.n_edges = n_edges;
  L.chunk = chunk ? chunk : generic ? pick_chunk_generic(n_edges) : pick_chunk(n_edges);
  DevBuf<uint32_t> deg(n, s), ntask(n, s);
  if (n) {
    ptr_degree_kernel<<<grid_for(n, 256), 256, 0, s>>>(kept_ptr, n, L.chunk, L.order.p, deg.p, ntask.p);
    UB_LAUNCH_CHECK();
  }
  DevBuf<uint32_t> dmax(1, s);
  reduce_max_u32(deg.p, n, dmax.p, s);
  DevBuf<uint64_t> tptr(n + 1, s);
  scan_u32_to_u64(ntask.p, tptr.p, n, s);
  uint64_t T = 0;
  UB_CUDA(cudaMemcpyAsync(&T, tptr.p + n, 8, cudaMemcpyDeviceToHost, s));
  UB_CUDA(cudaMemcpyAsync(&L.max_degree, dmax.p, 4, cudaMemcpyDeviceToHost, s));
  UB_CUDA(cudaStreamSynchronize(s));
  if (T >= 0xFFFFFFFFull) throw Error(UNSUPPORTED, "too many SGD tasks (>= 2^32)");
  L.n_tasks = T;
  DevBuf<uint32_t> trow(T, s), tkey(T, s), skey(T, s), perm(T, s);
  DevBuf<uint64_t> tstart(T, s);
  const int len_bits = bits_for(L.chunk);
  const uint32_t len_mask = (1u << len_bits) - 1u;
  const uint32_t n_seg = seg ? seg->n_seg : 0u;
  if ((uint64_t)n_seg << len_bits >= (1ull << 32)) throw Error(UNSUPPORTED, "too many instances for the task sort key");
  const int seg_bits = n_seg ? bits_for(n_seg) : 0;
  const bool renamed = L.order.p != nullptr;
  L.kernel = pick_epoch_kernel(n, dim, (T + 31) / 32, renamed, seg != nullptr, generic, alpha);
  L.block_threads = L.kernel == EpochKernel::Pool ? POOL_BT : 256;
  L.short_epoch = small_graph((T + 31) / 32);
  L.lane_major = lane_major_entries(n, seg != nullptr, L.kernel);
  TaskOrder torder = pick_task_order(renamed, L.short_epoch, seg != nullptr);
  if (torder == TaskOrder::LengthRate && len_bits + seg_bits + RATE_BITS > 32) torder = TaskOrder::Length;
  L.task_order = torder;
  const int rate_bits = torder == TaskOrder::LengthRate ? RATE_BITS : 0;
  int block_shift = -1, block_bits = 0;
  if (torder == TaskOrder::RowBlock) {
    block_shift = TASK_BLOCK_SHIFT;
    if (const char* e = getenv("UMAP_B200_TASK_BLOCK")) block_shift = std::min(31, std::max(0, atoi(e)));
    while (bits_for(n >> block_shift) + len_bits > 32) ++block_shift;  // the key fits 32 bits
    block_bits = bits_for(n >> block_shift);
  }
  if (n) {
    auto fill = [&](auto kernel, unsigned rows) {
      kernel<<<grid_for(n, rows), 256, 0, s>>>(kept_ptr, deg.p, tptr.p, n, L.chunk, seg ? seg->row_seg : nullptr,
                                               len_bits, rate_bits, block_shift, keps, L.order.p, trow.p, tstart.p,
                                               tkey.p);
      UB_LAUNCH_CHECK();
    };
    if (rate_bits) fill(task_fill_kernel<16>, 16);
    else fill(task_fill_kernel<1>, 256);
  }
  if (T && torder == TaskOrder::Row) {
    iota_u32_kernel<<<grid_for(T, 256), 256, 0, s>>>(perm.p, T);
    UB_LAUNCH_CHECK();
    UB_CUDA(cudaMemcpyAsync(skey.p, tkey.p, T * 4, cudaMemcpyDeviceToDevice, s));
  } else if (T) {
    radix_sort_pairs(tkey.p, nullptr, skey.p, perm.p, T, len_bits + (block_shift >= 0 ? block_bits : seg_bits) + rate_bits, s);
  }
  L.n_slices = (T + 31) / 32;
  L.slice_width.alloc(L.n_slices, s);
  L.split_mask.alloc(L.n_slices, s);
  L.rowid.alloc(L.n_slices * 32, s);
  L.slice_base.alloc(L.n_slices + 1, s);
  if (L.n_slices) {
    slice_meta_kernel<<<grid_for(L.n_slices * 32, 256), 256, 0, s>>>(perm.p, trow.p, skey.p, T, L.n_slices,
                                                                        L.chunk, rate_bits, len_mask, L.lane_major,
                                                                        L.slice_width.p, L.rowid.p,
                                                                        L.split_mask.p);
    UB_LAUNCH_CHECK();
  }
  DevBuf<uint64_t> wscan(L.n_slices + 1, s);
  scan_u32_to_u64(L.slice_width.p, wscan.p, L.n_slices, s);
  uint64_t wtot = 0;
  UB_CUDA(cudaMemcpyAsync(&wtot, wscan.p + L.n_slices, 8, cudaMemcpyDeviceToHost, s));
  UB_CUDA(cudaStreamSynchronize(s));
  L.n_entries = wtot * 32;
  L.entry.alloc(L.n_entries, s);
  if (L.n_slices) {
    slice_fill_kernel<<<grid_for(L.n_slices * 32 * (L.lane_major ? 8 : 1), 256), 256, 0, s>>>(ktail, keps, perm.p, tstart.p, skey.p, T,
                                                                        L.chunk, rate_bits, len_mask, wscan.p,
                                                                        L.slice_width.p, L.n_slices,
                                                                        L.lane_major, rank.p, L.entry.p);
    UB_LAUNCH_CHECK();
  }
  // slice_base = 32 * wscan (entries, not widths)
  scale32_kernel<<<grid_for(L.n_slices + 1, 256), 256, 0, s>>>(wscan.p, L.n_slices + 1);
  UB_LAUNCH_CHECK();
  UB_CUDA(cudaMemcpyAsync(L.slice_base.p, wscan.p, (L.n_slices + 1) * 8, cudaMemcpyDeviceToDevice, s));
  // count partial-row tasks (diagnostics)
  std::vector<uint32_t> h(L.n_slices);
  if (L.n_slices) UB_CUDA(cudaMemcpyAsync(h.data(), L.split_mask.p, L.n_slices * 4, cudaMemcpyDeviceToHost, s));
  UB_CUDA(cudaStreamSynchronize(s));
  L.split_tasks = 0;
  for (uint32_t v : h) L.split_tasks += __builtin_popcount(v);
}

void export_edges(const uint64_t* indptr, const uint32_t* indices, const float* data, uint64_t n,
                  float thr, float max_w, uint64_t total_epochs, const uint64_t* kept_ptr,
                  uint32_t* head, uint32_t* tail, double* eps, cudaStream_t s, const SegmentPrune* sp) {
  if (n == 0) return;
  export_edges_kernel<<<grid_for(n, 32), 256, 0, s>>>(
      indptr, indices, data, n, thr, (double)max_w, (double)total_epochs, sp ? sp->seg_thr : nullptr,
      sp ? sp->seg_maxw : nullptr, sp ? sp->row_seg : nullptr, kept_ptr, head, tail, eps);
  UB_LAUNCH_CHECK();
}

void normalize_init(float* emb, uint64_t n, uint32_t dim, cudaStream_t s, const Segments* seg) {
  if (n == 0 || dim == 0) return;
  const uint32_t n_seg = seg ? seg->n_seg : 1u;
  DevBuf<float> mins((uint64_t)dim * n_seg, s), scales((uint64_t)dim * n_seg, s);
  if (seg || dim > 65535) {  // batched instances: one block per (dimension, instance)
    minmax_dim_kernel<<<dim3(dim, n_seg), 1024, 0, s>>>(emb, n, dim, seg ? seg->seg_off : nullptr, mins.p, scales.p);
    UB_LAUNCH_CHECK();
  } else {
    const uint32_t G = (uint32_t)std::min<uint64_t>(256, (n + 4095) / 4096);
    DevBuf<float> pmin((uint64_t)dim * G, s), pmax((uint64_t)dim * G, s);
    minmax_part_kernel<<<dim3(G, dim), 256, 0, s>>>(emb, n, dim, pmin.p, pmax.p);
    UB_LAUNCH_CHECK();
    minmax_finish_kernel<<<dim, 32, 0, s>>>(pmin.p, pmax.p, G, mins.p, scales.p);
    UB_LAUNCH_CHECK();
  }
  normalize_kernel<<<grid_for(n * dim, 256), 256, 0, s>>>(emb, n * dim, dim, mins.p, scales.p,
                                                          seg ? seg->row_seg : nullptr);
  UB_LAUNCH_CHECK();
}

// Launches an epoch kernel; `overlap` makes it a programmatic dependent of the launch before it on
// the stream (only kernels that wait for that launch with grid_wait take it).
template <class... P, class... A>
void launch_epoch(void (*k)(P...), unsigned grid, unsigned bt, bool overlap, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(bt);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = overlap ? 1 : 0;
  UB_CUDA(cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...));
  count_launch();
}

// The launch may overlap the end of the epoch before it (`overlap`): the pooled kernel evaluates its
// schedule before grid_wait.  A large launch is released to the next one when its last blocks start, a
// smaller one at its blocks' end, since the next epoch's early blocks would fill the SMs unevenly
// (us per epoch, released at the end / early: 70k points 30.3 / 36.5, 300k (2,400 blocks) 84.0 / 85.2, 500k
// (3,900) 131.3 / 128.0, 1M 244.4 / 238.0, 2M 472.8 / 469.4).
constexpr unsigned EARLY_BLOCKS = 3500;
void sgd_epoch(const SgdLayout& L, float* live, float* snap, const SgdParams& p, uint32_t epoch, float alpha,
               bool overlap, cudaStream_t s) {
  if (L.n_slices == 0) return;
  constexpr unsigned BT = 256;
  const uint64_t tasks = L.n_slices * 32;
  auto blocks = [](uint64_t threads, unsigned bt) {
    const uint64_t g = (threads + bt - 1) / bt;
    if (g > 0x7FFFFFFFull) throw Error(UNSUPPORTED, "too many SGD tasks for one launch");
    return (unsigned)g;
  };
#define UB_SGD_ARGS L.slice_base.p, L.slice_width.p, L.split_mask.p, L.rowid.p, L.entry.p, L.n_slices, live, snap, \
                    p, epoch, alpha
  auto pooled = [&](auto k) {
    const unsigned g = blocks(tasks, POOL_BT);
    launch_epoch(k, g, POOL_BT, overlap, s, UB_SGD_ARGS, g > EARLY_BLOCKS);
  };
  const bool gen = p.generic_metric;
  auto variants = [&](auto dims) {  // dims(generic rule, batch)
    if (gen) p.row_seg ? dims(std::true_type{}, std::true_type{}) : dims(std::true_type{}, std::false_type{});
    else p.row_seg ? dims(std::false_type{}, std::true_type{}) : dims(std::false_type{}, std::false_type{});
  };
  switch (L.kernel) {
    case EpochKernel::Pool: {
      auto dims = [&](auto gen, auto seg) {
        constexpr bool G = gen.value, S = seg.value;
        auto many = [&](auto k, auto k_many) { pooled(!G && p.neg_rate >= (uint32_t)NB_POOL ? k_many : k); };
        if (p.dim == 1) many(sgd_epoch_pool<1, G, S, false>, sgd_epoch_pool<1, G, S, !G>);
        else if (p.dim == 2) many(sgd_epoch_pool<2, G, S, false>, sgd_epoch_pool<2, G, S, !G>);
        else if (p.dim == 3) many(sgd_epoch_pool<3, G, S, false>, sgd_epoch_pool<3, G, S, !G>);
        else many(sgd_epoch_pool<4, G, S, false>, sgd_epoch_pool<4, G, S, !G>);
      };
      variants(dims);
      break;
    }
    case EpochKernel::Lane: {
      const unsigned bt = L.block_threads;
      auto lanes = [&](auto k) { launch_epoch(k, blocks(tasks, bt), bt, false, s, UB_SGD_ARGS); };
      auto dims = [&](auto gen, auto seg, auto lm) {
        constexpr bool G = gen.value, S = seg.value, LM = lm.value;
        const bool eight = L.short_epoch && !G;
        if (p.dim == 1) lanes(eight ? sgd_epoch_kernel2<1, false, NB_SHORT, MINB_SHORT, LM, S> : sgd_epoch_kernel2<1, G, NB_WIDE, MINB_WIDE, LM, S>);
        else if (p.dim == 2) lanes(eight ? sgd_epoch_kernel2<2, false, NB_SHORT, MINB_SHORT, LM, S> : sgd_epoch_kernel2<2, G, NB_WIDE, MINB_WIDE, LM, S>);
        else if (p.dim == 3) lanes(sgd_epoch_kernel2<3, G, NB_WIDE, MINB_WIDE, LM, S>);
        else lanes(sgd_epoch_kernel2<4, G, NB_WIDE, MINB_WIDE, LM, S>);
      };
      if (L.lane_major) variants([&](auto gen, auto seg) { dims(gen, seg, std::true_type{}); });
      else if (gen) dims(std::true_type{}, std::false_type{}, std::false_type{});
      else dims(std::false_type{}, std::false_type{}, std::false_type{});
      break;
    }
    case EpochKernel::Rows:
      launch_epoch(p.dim == 5 ? sgd_epoch_rows<5> : p.dim == 6 ? sgd_epoch_rows<6> : sgd_epoch_rows<7>,
                   blocks(tasks, BT), BT, false, s, UB_SGD_ARGS);
      break;
    case EpochKernel::Dram:
      launch_epoch(p.dim == 1 ? sgd_epoch_dram<1> : sgd_epoch_dram<2>, blocks(tasks, BT), BT, false, s, UB_SGD_ARGS);
      break;
    case EpochKernel::AnyDim:
      launch_epoch(gen ? sgd_epoch_anydim<true> : sgd_epoch_anydim<false>, blocks(tasks, L.block_threads),
                   L.block_threads, false, s, UB_SGD_ARGS, L.lane_major);
      break;
  }
#undef UB_SGD_ARGS
}

void schedule_totals(const SgdLayout& L, uint32_t neg_rate, uint32_t start, uint32_t end,
                     unsigned long long* d_fired, unsigned long long* d_negs, cudaStream_t s) {
  UB_CUDA(cudaMemsetAsync(d_fired, 0, 8, s));
  UB_CUDA(cudaMemsetAsync(d_negs, 0, 8, s));
  if (L.n_entries == 0 || end <= start) return;
  schedule_totals_kernel<<<grid_for(L.n_entries, 256), 256, 0, s>>>(L.entry.p, L.n_entries, neg_rate, start, end,
                                                                   d_fired, d_negs);
  UB_LAUNCH_CHECK();
}

void negative_draws(uint64_t seed, uint64_t first, uint64_t count, uint32_t epoch, uint32_t per, uint32_t lo,
                    uint32_t range, uint32_t* out, cudaStream_t s) {
  if (count == 0 || per == 0) return;
  negative_draws_kernel<<<grid_for(count, 256), 256, 0, s>>>(seed, first, count, epoch, per, lo, range, out);
  UB_LAUNCH_CHECK();
}

void negatives_per_firing(const uint32_t* qs, const uint32_t* ns, uint64_t count, uint32_t neg, uint32_t* out,
                          cudaStream_t s) {
  if (count == 0) return;
  negatives_per_firing_kernel<<<grid_for(count, 256), 256, 0, s>>>(qs, ns, count, neg, out);
  UB_LAUNCH_CHECK();
}

void nan_empty_rows(const uint64_t* indptr, uint64_t n, uint32_t dim, float* emb, cudaStream_t s) {
  if (n == 0) return;
  nan_rows_kernel<<<grid_for(n, 256), 256, 0, s>>>(indptr, n, dim, emb);
  UB_LAUNCH_CHECK();
}

}  // namespace ub
