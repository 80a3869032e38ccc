// Exact k-nearest neighbours by brute force, the step before the fit path.  The reference
// takes kNN as input (umap-rs/src/lib.rs:41) and its example computes it by brute force
// (examples/src/bin/mnist_demo.rs:203-229): for every point the k others with the smallest
// Euclidean distance sqrt(sum_i (x_i - y_i)^2) (f32, summed in coordinate order), ordered by
// distance with ties in index order (a stable sort of the candidates 0..n), the point itself
// excluded; with fewer than k other points the missing slots stay zero.  This file returns
// exactly those arrays.
//
// Pipeline (one stream):
//  K-a  column means (f64 sums) and the largest centred magnitude, then per row: centred
//       values scaled by a power of two into the FP16 range and rounded to FP16 [n_pad, Dp]
//       (Dp = D rounded up to 64, zero padded), the squared norm of the rounded row, and the
//       f32 norm of the centred row (for the error bound).
//       From 16,384 points the rows are first put in locality order: each is assigned to the
//       nearest of 256 pivot rows (BF16 tensor-core GEMM) and the rows are sorted by pivot, so
//       a query block meets its neighbours in the first tiles it scans.
//  K-b  tensor-core candidate pass.  Persistent CTAs take (128 query rows, split) items and stream the
//       split's database tiles of 256 rows: warp 0 issues TMA loads (128-byte swizzle, 3 stages of a
//       128 x 64 query chunk and a 256 x 64 database chunk), warp 1 issues tcgen05.mma (M=128,
//       N=256, K=16, FP16, FP32 accumulation) into one of two 256-column tensor-memory
//       accumulators, and warps 2-9 read the other accumulator with tcgen05.ld (thread = query
//       row; warps 2-5 take the first 128 columns of a tile, warps 6-9 the rest).  For a dot
//       product s with database row y the approximate squared distance is |q|^2 + |y|^2 - 2s; the
//       epilogue tests s - |y|^2 / 2 against the row's threshold and appends the few entries
//       below it to its half's list of the row.  The two halves' lists of at most 32 are the
//       row's C = 64 candidates of the split, with their approximate distances.
//       The scan takes 16 tiles around the query block's own tile first, then the rest in the
//       order all CTAs share; the producer warp also bulk-copies each tile's row norms into a
//       ring of shared-memory slots.
//  K-c  exact rerank, a warp per row: the reference's f32 distance for each candidate whose
//       approximate distance leaves it a chance (the candidates' rows staged through shared memory
//       32 coordinates at a time, each lane summing its candidate's coordinates in order), the k
//       smallest (distance, index) pairs, and a certificate: any point that never entered the list has an approximate
//       squared distance >= tau, hence a true distance >= a lower bound that accounts for the
//       FP16 rounding of both rows, the accumulation error and the rounding of the
//       reference's own formula; if the k-th distance found is below that bound no outside
//       point can enter the top k.
//  K-d  rows whose certificate fails are recomputed exactly against all points: CTAs over
//       (row, column range) keep the k smallest keys of their range, then a warp per row
//       merges the ranges.  For k > 32 and fewer than 2,048 points every row takes this path.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "ub_internal.hpp"
#include "umma.cuh"

namespace ub {
namespace {

using namespace umma;

constexpr int QM = 128;      // query rows per CTA (UMMA M, tensor-memory lanes)
constexpr int DBN = 256;     // database rows per tile (UMMA N)
constexpr int KC = 64;       // K per staged chunk (128 bytes of bf16)
constexpr int TS = 3;        // pipeline stages
constexpr int NCAND = 64;    // candidates kept per row and database split
constexpr int HC = NCAND / 2;  // per epilogue warpgroup (each takes half of a tile's columns)
constexpr int CAP = 2 * HC;    // list slots per row and epilogue warpgroup
constexpr int KNN_THREADS = 320;
constexpr uint32_t Q_BYTES = QM * 128, D_BYTES = DBN * 128, STAGE = Q_BYTES + D_BYTES;
constexpr int NBS = 4;      // slots of the ring of per-tile row norms
constexpr size_t KNN_SMEM = (size_t)TS * STAGE + (size_t)2 * CAP * QM * 4 + NBS * DBN * 4 + 1024;
static_assert(STAGE % 1024 == 0, "stages stay 1024-byte aligned");
constexpr float PAD_NORM = 3.0e38f;  // |y|^2 of padding rows: never a candidate
constexpr uint64_t KNN_REORDER_MIN = 16384;  // scan in locality order from this many points

__device__ __forceinline__ uint64_t dist_key(float dist, uint32_t idx) {
  // non-negative floats order like their bit patterns: (distance, index) order in one u64
  return ((uint64_t)__float_as_uint(dist) << 32) | idx;
}

// ---------------------------------------------------------------------------- K-a
__global__ void col_sums_kernel(const float* __restrict__ X, int64_t n, int d, double* __restrict__ sums,
                                unsigned* __restrict__ cmin, unsigned* __restrict__ cmax,
                                unsigned* __restrict__ bad) {
  __shared__ double part[8][33];
  __shared__ float lo[8][33], hi[8][33];
  const int col = blockIdx.x * 32 + threadIdx.x;
  double acc = 0.0;
  float mn = INFINITY, mx = -INFINITY;
  bool finite = true;
  if (col < d)
    for (int64_t r = (int64_t)blockIdx.y * 8 + threadIdx.y; r < n; r += (int64_t)gridDim.y * 8) {
      const float v = X[r * d + col];
      finite &= isfinite(v);
      acc += (double)v;
      mn = fminf(mn, v);
      mx = fmaxf(mx, v);
    }
  if (!finite) atomicOr(bad, 1u);
  part[threadIdx.y][threadIdx.x] = acc;
  lo[threadIdx.y][threadIdx.x] = mn;
  hi[threadIdx.y][threadIdx.x] = mx;
  __syncthreads();
  if (threadIdx.y == 0 && col < d) {
    for (int i = 1; i < 8; ++i) {
      acc += part[i][threadIdx.x];
      mn = fminf(mn, lo[i][threadIdx.x]);
      mx = fmaxf(mx, hi[i][threadIdx.x]);
    }
    atomicAdd(sums + col, acc);
    // order-preserving integer images of the floats for atomicMin / atomicMax
    const unsigned umn = __float_as_uint(mn), umx = __float_as_uint(mx);
    atomicMin(cmin + col, (umn & 0x80000000u) ? ~umn : (umn | 0x80000000u));
    atomicMax(cmax + col, (umx & 0x80000000u) ? ~umx : (umx | 0x80000000u));
  }
}

__device__ __forceinline__ float from_ordered(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// Column means and the largest centred magnitude max_c max(max_c - mean_c, mean_c - min_c)
// (bit pattern of a non-negative float, atomicMax).
__global__ void col_means_kernel(const double* __restrict__ sums, const unsigned* __restrict__ cmin,
                                 const unsigned* __restrict__ cmax, int64_t n, int d, float* __restrict__ mean,
                                 unsigned* __restrict__ maxabs) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d) return;
  const float m = (float)(sums[c] / (double)n);
  mean[c] = m;
  const float a = fmaxf(fabsf(from_ordered(cmax[c]) - m), fabsf(m - from_ordered(cmin[c])));
  atomicMax(maxabs, __float_as_uint(a * (1.0f + 1e-6f)));
}

// One warp per output row r (source row src = perm ? perm[r] : r, rows >= n are padding):
// the centred row times `scale` rounded to FP16 (xh) and its squared norm (nb, scaled units),
// the same values rounded to BF16 (xb, for the pivot assignment), and the f32 norm of the
// centred row (rn, true units, rounded up slightly).  Null outputs are skipped.
__global__ void knn_prep_kernel(const float* __restrict__ X, int64_t n, int d, int dp, int64_t n_pad,
                                const float* __restrict__ mean, float scale, const uint32_t* __restrict__ perm,
                                __half* __restrict__ xh, float* __restrict__ nb, __nv_bfloat16* __restrict__ xb,
                                float* __restrict__ rn, unsigned* __restrict__ rmax_bits) {
  const int lane = threadIdx.x & 31;
  const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t r = w0; r < n_pad; r += nw) {
    const int64_t src = (r < n && perm) ? (int64_t)perm[r] : r;
    float s2 = 0.0f, sb = 0.0f;
    for (int c = lane; c < dp; c += 32) {
      float xc = 0.0f;
      if (r < n && c < d) xc = X[src * d + c] - mean[c];
      const __half h = __float2half_rn(xc * scale);
      const float hf = __half2float(h);
      if (xh) xh[r * dp + c] = h;
      if (xb) xb[r * dp + c] = __float2bfloat16_rn(xc * scale);
      s2 += xc * xc;
      sb += hf * hf;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      s2 += __shfl_xor_sync(0xFFFFFFFFu, s2, o);
      sb += __shfl_xor_sync(0xFFFFFFFFu, sb, o);
    }
    if (lane == 0) {
      if (nb) nb[r] = r < n ? sb : PAD_NORM;
      if (rn) {
        const float norm = r < n ? sqrtf(s2) * (1.0f + 1e-5f) : 0.0f;
        rn[src] = norm;
        atomicMax(rmax_bits, __float_as_uint(norm));
      }
    }
  }
}

// Locality order for the scan.  Pivot p is row p * n / P; its BF16 row and squared norm.
constexpr int NPIV = 256;
__global__ void gather_pivots_kernel(const __nv_bfloat16* __restrict__ xb, int64_t n, int dp,
                                     __nv_bfloat16* __restrict__ piv, float* __restrict__ pn) {
  const int p = blockIdx.x;
  const int64_t src = (int64_t)p * n / NPIV;
  float s = 0.0f;
  for (int c = threadIdx.x; c < dp; c += blockDim.x) {
    const __nv_bfloat16 v = xb[src * dp + c];
    piv[(int64_t)p * dp + c] = v;
    const float f = __bfloat162float(v);
    s += f * f;
  }
  __shared__ float red[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    pn[p] = s;
  }
}

// A warp per row of a chunk of x . p^T [rows, NPIV]: key = the nearest pivot (|p|^2 - 2 x.p).
__global__ void nearest_pivot_kernel(const float* __restrict__ dots, int64_t rows, int64_t row0, int64_t n,
                                     const float* __restrict__ pn, uint32_t* __restrict__ key) {
  const int lane = threadIdx.x & 31;
  const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (r >= rows || row0 + r >= n) return;
  float best = INFINITY;
  uint32_t arg = 0;
  for (int p = lane; p < NPIV; p += 32) {
    const float v = pn[p] - 2.0f * dots[r * NPIV + p];
    if (v < best) {
      best = v;
      arg = (uint32_t)p;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ob = __shfl_xor_sync(0xFFFFFFFFu, best, o);
    const uint32_t oa = __shfl_xor_sync(0xFFFFFFFFu, arg, o);
    if (ob < best || (ob == best && oa < arg)) {
      best = ob;
      arg = oa;
    }
  }
  if (lane == 0) key[row0 + r] = arg;
}

// tcgen05.ld of 32 consecutive accumulator columns of this warp's 32 lanes (thread = lane) and the
// wait for it; the wait's in-out operands keep every use of the registers behind it.
__device__ __forceinline__ void tmem_read(uint32_t (&r)[32], uint32_t taddr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                 "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                 "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

// The same of 16 columns.
__device__ __forceinline__ void tmem_read(uint32_t (&r)[16], uint32_t taddr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15])
               :
               : "memory");
}

// ---------------------------------------------------------------------------- K-b
// The list of one row and half: CAP slots, a bit of occ0 / occ1 per slot in use, its smallest entry so
// far in mn.  What bounds its size:
//  * k <= KNN_MAX_K: each half keeps its rank = ceil(k / 2) smallest distances in registers, in order
//    (RL of them, the first RL - rank at minus infinity).  With both halves' rank-th at or below y the
//    row's k-th smallest is at most y, and only entries under y plus the error margin can matter
//    (Margin): the threshold follows every hit.
//  * a list whose slots run out keeps what is at or below the threshold, and of that the HC smallest
//    (thin_list; the whole warp at once, a lane per list).  Longer k have only this (RL = 0), and keep
//    HC - 4 to HC, which is found sooner.
// Nothing moves: the slots of the others become free, and tau falls to a bound that no entry left
// out, now or later, is below.
struct Margin {
  float xr, R, gamma, scale, e2, rel;
  // approximate squared distance from which on a point's lower bound exceeds the upper bound of one at a
  __device__ __forceinline__ float beyond(float a) const {
    const float inv = 1.0f / scale, s = 1.001f * (xr + R), e1 = gamma * s * s;
    const float u = sqrtf(fmaxf(0.0f, a * inv * inv) + e1) + e2;
    return (u * u * rel + e1) * scale * scale;
  }
};
// By value: a list's words must not be given an address, or they would live in local memory, which
// the little L1 beside this kernel's shared memory does not hold.
struct ListState {
  uint32_t occ0, occ1;
  float tau;
};
__device__ __noinline__ ListState thin_list(const float* ld, uint32_t occ0, uint32_t occ1, float tau, float mn, int keep) {
  float e[CAP];  // free slots count as infinite
#pragma unroll
  for (int j = 0; j < CAP; ++j) {
    const float x = ld[j * QM];
    e[j] = ((j < 32 ? occ0 : occ1) >> (j & 31)) & 1u ? x : INFINITY;
  }
  auto at_most = [&](float v) {
    int c = 0;
#pragma unroll
    for (int j = 0; j < CAP; ++j) c += e[j] <= v ? 1 : 0;
    return c;
  };
  float top = tau;  // every entry is below it
  if (!(top < INFINITY)) {
    top = -INFINITY;
#pragma unroll
    for (int j = 0; j < CAP; ++j) top = fmaxf(top, e[j] < INFINITY ? e[j] : -INFINITY);
  }
  // h with at_most(h) in [lo_count, hi_count] where there is one: interpolation on the counts, then
  // bisection; every lane of the warp runs it, those with `go` unset only along
  auto search = [&](bool go, int lo_count, int hi_count, float& l, float h, int ch) {
    int cl = 0;  // at_most(l) < lo_count, or l is the smallest entry
    for (int it = 0; it < 28; ++it) {
      const float f = it < 6 && (it & 1) == 0 ? ((float)(lo_count - cl) + 0.5f) / (float)(ch - cl) : 0.5f;
      const float mid = l + (h - l) * f;
      go = go && ch > hi_count && mid > l && mid < h;
      if (!__any_sync(0xFFFFFFFFu, go)) break;
      const int c = at_most(mid);
      if (go) {
        if (c >= lo_count) {
          h = mid;
          ch = c;
        } else {
          l = mid;
          cl = c;
        }
      }
    }
    return h;
  };
  float t = top;
  const int have = at_most(t);
  float l = mn;
  const bool cut = have > HC;
  if (__any_sync(0xFFFFFFFFu, cut)) {
    const float x = search(cut, keep, HC, l, top, have);
    if (cut) t = x;
  }
  uint32_t m0 = 0, m1 = 0;
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    m0 |= e[j] <= t ? 1u << j : 0u;
    m1 |= e[j + 32] <= t ? 1u << j : 0u;
  }
  if (__popc(m0) + __popc(m1) > HC) {  // ties above l: as many as fit
    uint32_t x0 = 0, x1 = 0;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      x0 |= e[j] < l ? 1u << j : 0u;
      x1 |= e[j + 32] < l ? 1u << j : 0u;
    }
    uint32_t y0 = m0 & ~x0, y1 = m1 & ~x1;
    for (int room = HC - __popc(x0) - __popc(x1); room > 0; --room) {
      if (y0) {
        x0 |= y0 & (0u - y0);
        y0 &= y0 - 1;
      } else {
        x1 |= y1 & (0u - y1);
        y1 &= y1 - 1;
      }
    }
    m0 = x0;
    m1 = x1;
    t = l;  // what was left out is at l or above
  }
  return ListState{m0, m1, cut || t < top ? fminf(tau, t) : tau};
}

// Persistent: CTA b takes the work items b, b + gridDim.x, ... of q_blocks x n_splits (query block,
// split); split s scans the tiles s, s + n_splits, ...  The query blocks are the q_blocks from q_first on, and the
// candidate arrays hold their rows only, in scan order.
template <int RL>
__global__ void __launch_bounds__(KNN_THREADS, 1) knn_candidates_kernel(
    const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tdb, const float* __restrict__ nb,
    int64_t n, int n_kchunks, int64_t tiles_total, int64_t q_first, int64_t q_blocks, int n_splits, int k, int d,
    const unsigned* __restrict__ rmax_bits, float gamma, float scale, const uint32_t* __restrict__ perm,
    uint32_t* __restrict__ list_idx, uint32_t* __restrict__ cand_idx, float* __restrict__ cand_d,
    float* __restrict__ tau_out, unsigned* __restrict__ err) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full[TS], empty[TS], tfull[2], tempty[2], nfull[NBS], nempty[NBS];
  __shared__ uint32_t tmem_base;
  __shared__ volatile int s_fail;
  // [item % 4][half][row]: the half's rank-th smallest, infinite until there is one (the halves are at
  // most two tiles apart, so two items)
  __shared__ float s_rank[4][2][QM];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  float* lists = reinterpret_cast<float*>(smem + TS * STAGE);  // [2][CAP][QM] approximate distances of the halves' lists
  float* nbuf = lists + 2 * CAP * QM;                          // [NBS][DBN] norms of the tile's rows
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t items = q_blocks * n_splits;
  // An item's scan order: first a window of WIN tiles around the query block's own tile (rows in
  // locality order: its nearest neighbours come first and the candidate threshold tightens
  // early), then the rest in increasing order, which all CTAs share, so the CTAs resident
  // together read the same tiles and the database streams through L2 once per wave.
  constexpr int64_t WIN = 16;
  struct Item {
    int64_t m0, w0;
    int split, T, wn, S;
    __device__ __forceinline__ Item(int64_t w, int64_t q_first, int64_t q_blocks, int n_splits, int64_t tiles) {
      split = (int)(w / q_blocks);
      S = n_splits;
      m0 = (q_first + w - (int64_t)split * q_blocks) * QM;
      T = (int)((tiles - split + n_splits - 1) / n_splits);
      int64_t own = m0 / DBN / n_splits - WIN / 2;
      own = own < 0 ? 0 : own;
      own = own > T - WIN ? T - WIN : own;
      w0 = T > WIN ? own : 0;
      wn = T > WIN ? (int)WIN : 0;
    }
    __device__ __forceinline__ int64_t tile(int t) const {
      const int64_t u = t < wn ? w0 + t : (t - wn < w0 ? (int64_t)(t - wn) : (int64_t)t);
      return split + u * S;
    }
  };

  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&tmem_base)), "r"(2 * DBN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < TS; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&full[i])), "r"(1) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&empty[i])), "r"(1) : "memory");
    }
    for (int i = 0; i < 2; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&tfull[i])), "r"(1) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&tempty[i])), "r"(2 * QM) : "memory");
    }
    for (int i = 0; i < NBS; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&nfull[i])), "r"(1) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(&nempty[i])), "r"(2 * QM) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_fail = 0;
  }
  for (int i = tid; i < 4 * 2 * QM; i += KNN_THREADS) (&s_rank[0][0][0])[i] = INFINITY;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tbase = tmem_base;

  // g counts staged chunks and tt tiles over all of the CTA's items: the barriers' phases run on
  if (warp == 0) {
    if (lane == 0) {  // TMA producer
      int64_t g = 0, tt = 0, n_issued = 0;
      bool ok = true;
      for (int64_t w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const Item it(w, q_first, q_blocks, n_splits, tiles_total);
        for (int t = 0; t < it.T && ok; ++t, ++tt) {
          const int64_t tile = it.tile(t);
          for (int c = 0; c < n_kchunks; ++c, ++g) {
            const int st = (int)(g % TS);
            if (s_fail || (g >= TS && !mbar_wait(smem_u32(&empty[st]), (uint32_t)(((g / TS) - 1) & 1)))) {
              ok = false;
              break;
            }
            if (c == 0) {
              // the tile's row norms go to slot tt % NBS once the epilogue is done with tile tt - NBS
              const int slot = (int)(tt % NBS);
              if (tt >= NBS && !mbar_wait(smem_u32(&nempty[slot]), (uint32_t)(((tt / NBS) - 1) & 1))) {
                ok = false;
                break;
              }
              const uint32_t nfb = smem_u32(&nfull[slot]);
              asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(nfb), "r"(DBN * 4) : "memory");
              asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                           :: "r"(smem_u32(nbuf + slot * DBN)), "l"(nb + tile * DBN), "r"(DBN * 4), "r"(nfb)
                           : "memory");
              n_issued = tt + 1;
            }
            const uint32_t q_dst = smem_u32(smem + st * STAGE), d_dst = q_dst + Q_BYTES;
            const uint32_t fb = smem_u32(&full[st]);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(fb), "r"(STAGE) : "memory");
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                :: "r"(q_dst), "l"(reinterpret_cast<uint64_t>(&tq)), "r"(c * KC), "r"((int)it.m0), "r"(fb) : "memory");
            asm volatile(
                "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                :: "r"(d_dst), "l"(reinterpret_cast<uint64_t>(&tdb)), "r"(c * KC), "r"((int)(tile * DBN)),
                   "r"(fb) : "memory");
          }
        }
      }
      if (!ok) s_fail = 1;
      // the copies of the last stages and norm buffers must have landed before the CTA may exit
      for (int64_t h = g > TS ? g - TS : 0; h < g; ++h) (void)mbar_wait(smem_u32(&full[h % TS]), (uint32_t)((h / TS) & 1));
      for (int64_t t = n_issued > NBS ? n_issued - NBS : 0; t < n_issued; ++t)
        (void)mbar_wait(smem_u32(&nfull[t % NBS]), (uint32_t)((t / NBS) & 1));
    }
  } else if (warp == 1) {
    if (lane == 0) {  // MMA issuer
      constexpr uint32_t idesc = instr_desc_f16(QM, DBN);
      int64_t g = 0, tt = 0;
      bool ok = true;
      for (int64_t w = blockIdx.x; w < items && ok; w += gridDim.x) {
        const int T = Item(w, q_first, q_blocks, n_splits, tiles_total).T;
        for (int t = 0; t < T && ok; ++t, ++tt) {
          const int buf = (int)(tt & 1);
          if (tt >= 2 && !mbar_wait(smem_u32(&tempty[buf]), (uint32_t)(((tt >> 1) - 1) & 1))) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t dacc = tbase + (uint32_t)(buf * DBN);
          for (int c = 0; c < n_kchunks; ++c) {
            const int st = (int)(g % TS);
            if (s_fail || !mbar_wait(smem_u32(&full[st]), (uint32_t)((g / TS) & 1))) {
              ok = false;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a0 = smem_u32(smem + st * STAGE), b0 = a0 + Q_BYTES;
#pragma unroll
            for (int k = 0; k < KC / 16; ++k) {
              const uint64_t ad = smem_desc_sw128(a0 + k * 32), bd = smem_desc_sw128(b0 + k * 32);
              const uint32_t acc = (c > 0 || k > 0) ? 1u : 0u;
              asm volatile(
                  "{\n\t.reg .pred p;\n\t"
                  "setp.ne.b32 p, %4, 0;\n\t"
                  "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
                  :: "r"(dacc), "l"(ad), "l"(bd), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
                  : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         :: "r"(smem_u32(&empty[st])) : "memory");
            ++g;
          }
          if (!ok) break;
          asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                       :: "r"(smem_u32(&tfull[buf])) : "memory");
        }
      }
      if (!ok) s_fail = 1;
      // the last MMAs must have completed before tensor memory is freed
      if (g > 0) (void)mbar_wait(smem_u32(&empty[(g - 1) % TS]), (uint32_t)(((g - 1) / TS) & 1));
    }
  } else {
    // epilogue: warps 2..9; warp w owns tensor-memory lane quarter w % 4 (query rows) and half
    // (w - 2) / 4 of each tile's columns, with its own list per row: entries below the row's
    // threshold go to free slots, and a list that runs out of them is reduced to its HC smallest
    // (thin_list), which lowers the threshold.
    const int q = warp & 3, half = (warp - 2) >> 2;
    const int trow = q * 32 + lane;
    float* ld = lists + half * CAP * QM + trow;
    const uint32_t ld_addr = smem_u32(ld);
    uint32_t* li = list_idx + ((int64_t)blockIdx.x * 2 + half) * CAP * QM + trow;
    // columns taken up at a time: 32, or 16 beside the longer ranked list (no register to spill)
    constexpr int COLS = RL > 8 ? 16 : 32;
    const int rank = (k + 1) / 2;  // at most RL, if RL
    Margin mg;
    mg.R = __uint_as_float(*rmax_bits);
    mg.gamma = gamma;
    mg.scale = scale;
    mg.rel = 1.0f + (float)(d + 16) * 8.0e-7f;
    int64_t tt = 0;
    int slot4 = 0;
    bool ok = true;
    for (int64_t w = blockIdx.x; w < items && ok; w += gridDim.x, slot4 = (slot4 + 1) & 3) {
      const Item it(w, q_first, q_blocks, n_splits, tiles_total);
      const int64_t row = it.m0 + trow;
      const bool live = row < n;
      const float nq = live ? nb[row] : 0.0f;
      uint32_t occ0 = 0, occ1 = 0;
      // thr = (|q|^2 - tau) / 2; padding columns (u = s - PAD_NORM / 2) stay below the first one
      float tau = INFINITY, thr = live ? -1.0e37f : INFINITY;
      mg.xr = sqrtf(fmaxf(nq, 0.0f)) / scale;
      mg.e2 = 2.0f * (0.00048876f * (mg.xr + mg.R) + 2.0f * sqrtf((float)(n_kchunks * KC)) * 2.9802322e-8f / scale);
      volatile float* mine = &s_rank[slot4][half][q * 32];
      const volatile float* other = &s_rank[slot4][half ^ 1][q * 32];
      float mn = INFINITY;  // the list's smallest entry so far
      float best[RL ? RL : 1];
#pragma unroll
      for (int i = 0; i < RL; ++i) best[i] = i < RL - rank ? -INFINITY : INFINITY;
      auto thin = [&]() {
        const ListState st = thin_list(ld, occ0, occ1, tau, mn, RL ? HC : HC - 4);
        occ0 = st.occ0;
        occ1 = st.occ1;
        tau = st.tau;
        if (live) thr = fmaxf(thr, 0.5f * (nq - tau));
      };
      // u = s - |y|^2 / 2 (half of 2 s - |y|^2 exactly) of 4 columns, two per packed FMA; a column
      // enters the list when |q|^2 - 2 u < tau, i.e. u > thr
      auto half_dist4 = [](float (&v)[4], const uint32_t* r, const float* nrm) {
        const uint64_t mhalf = 0xBF000000BF000000ull;  // (-0.5f, -0.5f)
        const float4 y = *reinterpret_cast<const float4*>(nrm);
        uint64_t s0, s1, n0, n1, d0, d1;
        asm("mov.b64 %0, {%1, %2};" : "=l"(s0) : "r"(r[0]), "r"(r[1]));
        asm("mov.b64 %0, {%1, %2};" : "=l"(s1) : "r"(r[2]), "r"(r[3]));
        asm("mov.b64 %0, {%1, %2};" : "=l"(n0) : "r"(__float_as_uint(y.x)), "r"(__float_as_uint(y.y)));
        asm("mov.b64 %0, {%1, %2};" : "=l"(n1) : "r"(__float_as_uint(y.z)), "r"(__float_as_uint(y.w)));
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d0) : "l"(n0), "l"(mhalf), "l"(s0));
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d1) : "l"(n1), "l"(mhalf), "l"(s1));
        uint32_t a0, a1, a2, a3;
        asm("mov.b64 {%0, %1}, %2;" : "=r"(a0), "=r"(a1) : "l"(d0));
        asm("mov.b64 {%0, %1}, %2;" : "=r"(a2), "=r"(a3) : "l"(d1));
        v[0] = __uint_as_float(a0);
        v[1] = __uint_as_float(a1);
        v[2] = __uint_as_float(a2);
        v[3] = __uint_as_float(a3);
      };
      // enters the columns c0 .. c0 + 7
      auto process = [&](const uint32_t* r, const float* nrm, int64_t c0) {
        float v[8], gm = -INFINITY;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float w4[4];
          half_dist4(w4, r + 4 * i, nrm + 4 * i);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            v[4 * i + j] = w4[j];
            gm = fmaxf(gm, w4[j]);
          }
        }
        if (!__any_sync(0xFFFFFFFFu, gm > thr)) return;
        if (c0 < it.m0 + QM && c0 + 8 > it.m0) {  // the columns may hold the row itself
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (c0 + i == row) v[i] = -INFINITY;
        }
        const bool low = __popc(occ0) <= 24;
        uint32_t free = ~(low ? occ0 : occ1);
        const uint32_t dst = ld_addr + (low ? 0u : 32u * QM * 4u);
        uint32_t* ids = li + (low ? 0 : 32 * QM);
        // a predicated append (no branch: some lane hits, most do not)
        auto append = [&](bool hit, float u, uint32_t col) {
          const uint32_t slot = (uint32_t)__ffs(free) - 1u;
          const float x = hit ? nq - 2.0f * u : INFINITY;
          asm volatile(
              "{\n\t.reg .pred p;\n\t"
              "setp.ne.u32 p, %0, 0;\n\t"
              "@p st.shared.f32 [%1], %2;\n\t"
              "@p st.global.u32 [%3], %4;\n\t}"
              :: "r"((uint32_t)hit), "r"(dst + slot * (QM * 4)), "f"(x), "l"(ids + slot * QM), "r"(col)
              : "memory");
          mn = fminf(mn, x);
          free = hit ? free & (free - 1u) : free;
          float y = x;
#pragma unroll
          for (int i = 0; i < RL; ++i) {  // into its place among the RL smallest
            const float b = best[i];
            best[i] = fminf(b, y);
            y = fmaxf(b, y);
          }
        };
        uint32_t hits = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) hits |= v[i] > thr ? 1u << i : 0u;
        if (__any_sync(0xFFFFFFFFu, __popc(hits) > 2)) {
#pragma unroll
          for (int i = 0; i < 8; ++i) append((hits >> i) & 1u, v[i], (uint32_t)c0 + i);
        } else {
          do {
            const int i = __ffs(hits) - 1;
            const float x0 = (i & 1) ? v[1] : v[0], x1 = (i & 1) ? v[3] : v[2];
            const float x2 = (i & 1) ? v[5] : v[4], x3 = (i & 1) ? v[7] : v[6];
            append(hits != 0, (i & 4) ? ((i & 2) ? x3 : x2) : ((i & 2) ? x1 : x0), (uint32_t)c0 + i);
            hits &= hits - 1;
          } while (__any_sync(0xFFFFFFFFu, hits != 0));
        }
        occ0 = low ? ~free : occ0;
        occ1 = low ? occ1 : ~free;
        if constexpr (RL > 0) {
          const float own = best[RL - 1];
          mine[lane] = own;
          const float y = fmaxf(own, other[lane]);
          if (y < INFINITY) {
            tau = fminf(tau, mg.beyond(y));
            if (live) thr = fmaxf(thr, 0.5f * (nq - tau));
          }
        }
      };
      for (int t = 0; t < it.T; ++t, ++tt) {
        const int buf = (int)(tt & 1);
        const int slot = (int)(tt % NBS);
        if (!mbar_wait(smem_u32(&tfull[buf]), (uint32_t)((tt >> 1) & 1)) ||
            !mbar_wait(smem_u32(&nfull[slot]), (uint32_t)((tt / NBS) & 1)) || s_fail) {
          s_fail = 1;
        }
        // one lane's failure ends the warp together
        if (__any_sync(0xFFFFFFFFu, s_fail != 0)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const int64_t cb0 = it.tile(t) * DBN + half * (DBN / 2);
        const float* nrm = nbuf + slot * DBN + half * (DBN / 2);
        const uint32_t ta = tbase + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * DBN + half * (DBN / 2));
#pragma unroll 1
        for (int jj = 0; jj < DBN / 2; jj += COLS) {
          uint32_t ra[COLS];
          tmem_read(ra, ta + (uint32_t)jj);
          const float* nj = nrm + jj;
          // the largest u of the chunk decides for the whole warp; only a chunk with an entry for
          // some row takes the columns up again, 8 at a time
          float gm = -INFINITY;
#pragma unroll
          for (int i = 0; i < COLS / 4; ++i) {
            float v[4];
            half_dist4(v, ra + 4 * i, nj + 4 * i);
            gm = fmaxf(gm, fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3])));
          }
          if (__any_sync(0xFFFFFFFFu, gm > thr)) {
#pragma unroll
            for (int h = 0; h < COLS / 8; ++h) {
              // 8 free slots in one of the list's halves, or the lists are thinned first.  The columns are
              // read again after the call: live across it they would be spilled, to L2
              if (__any_sync(0xFFFFFFFFu, __popc(occ0) > 24 && __popc(occ1) > 24)) {
                thin();
                tmem_read(ra, ta + (uint32_t)jj);
              }
              process(ra + 8 * h, nj + 8 * h, cb0 + jj + 8 * h);
            }
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(&tempty[buf])) : "memory");
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(smem_u32(&nempty[slot])) : "memory");
      }
      if (!ok) break;
      thin();
      mine[lane] = INFINITY;
      if (live) {  // candidates as original indices
        const int64_t at = (row - q_first * QM) * n_splits + it.split, base = at * NCAND + half * HC;
        for (int s = 0; s < HC; ++s) {
          const bool low = occ0 != 0, any = low || occ1 != 0;
          const int slot = low ? __ffs(occ0) - 1 : __ffs(occ1) + 31;
          if (low) occ0 &= occ0 - 1;
          else occ1 &= occ1 - 1;
          const uint32_t c = any ? li[slot * QM] : 0xFFFFFFFFu;
          cand_idx[base + s] = (perm && any) ? perm[c] : c;
          cand_d[base + s] = any ? ld[slot * QM] : INFINITY;
        }
        tau_out[at * 2 + half] = tau;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (tid == 0 && s_fail) atomicOr(err, 1u);
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tbase), "r"(2 * DBN) : "memory");
}

// ---------------------------------------------------------------------------- K-c
// Lower bound on the reference's distance from row x to any point y whose approximate squared
// distance (scaled units) is >= tau.  With x~, y~ the centred rows (|y~| <= R), x^, y^ their
// FP16 roundings after scaling by `scale` (a power of two):
//   |approx - |x^ - y^|^2| <= gamma (|x^| + |y^|)^2        (FP32 accumulation of the products
//                                                          and of the norms; generous)
//   | |x^ - y^| / scale - |x - y| | <= 2^-11 (1 + 2^-10) (|x~| + |y~|) + 2 sqrt(Dp) 2^-25 / scale
//                                                          (rounding to FP16 incl. subnormals,
//                                                          and the centring)
//   ref(x, y) >= |x - y| (1 - (D + 8) 2^-23)               (the reference's own f32 formula)
__device__ __forceinline__ float distance_lower_bound(float tau, float xr, float R, float gamma, float scale,
                                                      int d, int dp) {
  const float inv = 1.0f / scale;
  const float s = 1.001f * (xr + R);
  const float e1 = gamma * s * s;
  const float lb = sqrtf(fmaxf(0.0f, tau * inv * inv - e1)) - 0.00048876f * (xr + R) -
                   2.0f * sqrtf((float)dp) * 2.9802322e-8f * inv;
  return lb * (1.0f - (float)(d + 8) * 1.1920929e-7f) * (1.0f - 1e-6f);
}

// Upper bound on the reference's distance to a point whose approximate squared distance (scaled
// units) is at most a: the same error terms, added.
__device__ __forceinline__ float distance_upper_bound(float a, float xr, float R, float gamma, float scale, int d,
                                                      int dp) {
  const float inv = 1.0f / scale;
  const float s = 1.001f * (xr + R);
  const float ub = sqrtf(fmaxf(0.0f, a * inv * inv) + gamma * s * s) + 0.00048876f * (xr + R) +
                   2.0f * sqrtf((float)dp) * 2.9802322e-8f * inv;
  return ub * (1.0f + (float)(d + 8) * 1.1920929e-7f) * (1.0f + 1e-6f);
}

// The reference's distances from row x to m <= 32 rows (one per lane): the warp stages the rows
// 32 coordinates at a time in shared memory (coalesced 128-byte reads) and each lane sums its
// row's squared differences in coordinate order.
__device__ __forceinline__ float ref_distance_warp(const float* __restrict__ X, int d, int64_t row, uint32_t mine, int m,
                                                   float (*tile)[33], int lane) {
  float acc = 0.0f;
  for (int i0 = 0; i0 < d; i0 += 32) {
    const int i = i0 + lane;
#pragma unroll 8
    for (int j = 0; j < m; ++j) {
      const uint32_t c = __shfl_sync(0xFFFFFFFFu, mine, j);
      tile[j][lane] = i < d ? __ldg(X + (int64_t)c * d + i) : 0.0f;
    }
    tile[32][lane] = i < d ? __ldg(X + row * d + i) : 0.0f;
    __syncwarp();
    const int w = min(32, d - i0);
    for (int t = 0; t < w; ++t) {
      const float df = __fsub_rn(tile[32][t], tile[lane][t]);
      acc = __fadd_rn(acc, __fmul_rn(df, df));
    }
    __syncwarp();
  }
  return __fsqrt_rn(acc);
}

// Only candidates that can be among the k nearest are evaluated: with U the upper bound of (about)
// the k-th smallest approximate distance, at least k candidates' reference distances are at most
// U, and one whose lower bound is above U has k nearer ones.  On 70,000 x 784 images about 20 of
// the 64 are left.
constexpr int RERANK_BT = 128;
template <int E>  // candidates per lane = splits * NCAND / 32
__global__ void __launch_bounds__(RERANK_BT) knn_rerank_kernel(
    const float* __restrict__ X, int64_t n, int64_t first, int64_t count, int d, int dp, int k,
    const uint32_t* __restrict__ cand_idx,
    const float* __restrict__ cand_d, const float* __restrict__ tau_in, const float* __restrict__ rn,
    const unsigned* __restrict__ rmax_bits, float gamma, float scale, const uint32_t* __restrict__ order,
    uint32_t* __restrict__ out_idx, float* __restrict__ out_d, uint32_t* __restrict__ fail_rows,
    unsigned* __restrict__ fail_count) {
  constexpr int S = E * 32 / NCAND;
  __shared__ float tiles[RERANK_BT / 32][33][33];
  __shared__ uint32_t picked[RERANK_BT / 32][E * 32];
  const int lane = threadIdx.x & 31;
  float (*tile)[33] = tiles[threadIdx.x >> 5];
  uint32_t* pick = picked[threadIdx.x >> 5];
  for (int j = 0; j < 33; ++j) tile[j][lane] = 0.0f;
  const float R = __uint_as_float(*rmax_bits);
  const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t w = w0; w < count; w += nw) {
    // rows in locality order when there is one: neighbouring warps share candidate rows in L2
    const int64_t row = order ? (int64_t)order[first + w] : first + w;
    const float xr = rn[row];
    uint32_t ci[E];
    float ca[E], lo = INFINITY, hi = -INFINITY;
    int have = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      ci[e] = cand_idx[w * (S * NCAND) + e * 32 + lane];
      const bool valid = ci[e] < (uint64_t)n;
      ca[e] = valid ? cand_d[w * (S * NCAND) + e * 32 + lane] : INFINITY;
      if (valid) {
        lo = fminf(lo, ca[e]);
        hi = fmaxf(hi, ca[e]);
      }
      have += __popc(__ballot_sync(0xFFFFFFFFu, valid));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
    }
    float tau = lane < 2 * S ? tau_in[w * 2 * S + lane] : INFINITY;  // (split, half)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tau = fminf(tau, __shfl_xor_sync(0xFFFFFFFFu, tau, o));
    const float lb = tau < INFINITY ? distance_lower_bound(tau, xr, R, gamma, scale, d, dp) : INFINITY;
    float U = INFINITY;
    if (have > k) {
      // hi: at least k candidates at or below it, close to the k-th
      for (int it = 0; it < 24; ++it) {
        const float mid = 0.5f * (lo + hi);
        if (!(mid > lo && mid < hi)) break;
        int c = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) c += __popc(__ballot_sync(0xFFFFFFFFu, ca[e] <= mid));
        if (c >= k) {
          hi = mid;
          if (c <= k + 1) break;
        } else {
          lo = mid;
        }
      }
      // The k-th approximate distance, above lo, is at the certificate's bound or beyond: the exact one, which
      // the bound's margins stand far from, will not pass either, and the row is not worth evaluating
      // (3,000 x 784 of very uneven lengths, k = 128, all rows failing: 24.7 -> 23.0 ms a call).
      if (sqrtf(fmaxf(lo, 0.0f)) / scale >= lb) {
        if (lane == 0) fail_rows[atomicAdd(fail_count, 1u)] = (uint32_t)row;
        continue;
      }
      U = distance_upper_bound(hi, xr, R, gamma, scale, d, dp);
    }
    int m = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const bool want = ci[e] < (uint64_t)n && !(distance_lower_bound(ca[e], xr, R, gamma, scale, d, dp) > U);
      const unsigned b = __ballot_sync(0xFFFFFFFFu, want);
      if (want) pick[m + __popc(b & ((1u << lane) - 1u))] = ci[e];
      m += __popc(b);
    }
    __syncwarp();
    uint64_t keys[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      keys[e] = ~0ull;
      if (e * 32 < m) {
        const int left = min(32, m - e * 32);
        const uint32_t c = lane < left ? pick[e * 32 + lane] : 0u;
        const float dist = ref_distance_warp(X, d, row, c, left, tile, lane);
        if (lane < left) keys[e] = dist_key(dist, c);
      }
    }
    __syncwarp();
    uint64_t last = ~0ull;
    for (int p = 0; p < k; ++p) {
      uint64_t mn = ~0ull;
#pragma unroll
      for (int e = 0; e < E; ++e) mn = keys[e] < mn ? keys[e] : mn;
      uint64_t wm = mn;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const uint64_t other = __shfl_xor_sync(0xFFFFFFFFu, wm, o);
        wm = other < wm ? other : wm;
      }
      if (wm != ~0ull && mn == wm) {  // keys are distinct (distinct indices): one lane owns it
#pragma unroll
        for (int e = 0; e < E; ++e)
          if (keys[e] == wm) keys[e] = ~0ull;
      }
      if (lane == 0) {
        out_idx[row * k + p] = wm == ~0ull ? 0u : (uint32_t)wm;
        out_d[row * k + p] = wm == ~0ull ? 0.0f : __uint_as_float((uint32_t)(wm >> 32));
      }
      last = wm;
    }
    if (lane == 0 && tau < INFINITY && (last == ~0ull || !(__uint_as_float((uint32_t)(last >> 32)) < lb)))
      fail_rows[atomicAdd(fail_count, 1u)] = (uint32_t)row;
  }
}

// ---------------------------------------------------------------------------- K-d
// Exact brute force for the listed rows.  CTA (b, s) takes row rows[b] against the columns of
// range s: tiles of 256 columns are staged 32 coordinates at a time in shared memory
// (coalesced), each thread sums its column's squared differences in coordinate order and
// keeps its k smallest (distance, index) keys; k rounds of a block-wide minimum leave the
// range's k smallest keys in part[b][s][0..k).
// TH threads per CTA: 256 for k <= 32, 128 for the longer lists of k <= 128.
template <int TH>
__global__ void __launch_bounds__(TH) knn_exact_part_kernel(const float* __restrict__ X, int64_t n, int d, int k,
                                                            const uint32_t* __restrict__ rows, unsigned n_rows,
                                                            int n_ranges, uint64_t* __restrict__ part) {
  constexpr int EX_THREADS = TH, NW = TH / 32;
  extern __shared__ uint64_t lst[];  // [k][EX_THREADS]
  __shared__ float xt[32][EX_THREADS + 1];
  __shared__ float xs[32];
  __shared__ uint64_t red[EX_THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int s = blockIdx.y;
  const int64_t j_begin = n * s / n_ranges, j_end = n * (s + 1) / n_ranges;
  for (unsigned b = blockIdx.x; b < n_rows; b += gridDim.x) {
    const int64_t row = rows[b];
    for (int t = 0; t < k; ++t) lst[t * EX_THREADS + tid] = ~0ull;
    uint64_t mx = ~0ull;
    int ms = 0;
    for (int64_t j0 = j_begin; j0 < j_end; j0 += EX_THREADS) {
      const int64_t j = j0 + tid;
      float acc = 0.0f;
      for (int i0 = 0; i0 < d; i0 += 32) {
        __syncthreads();
        // 256 columns x 32 coordinates: warp w loads rows j0 + 32 w' .. as 128-byte pieces
        float ld[32];  // this warp's 32 rows: all loads in flight before the stores
#pragma unroll
        for (int u = 0; u < 32; ++u) {
          const int64_t jj = j0 + warp + NW * u;
          ld[u] = (jj < j_end && i0 + lane < d) ? __ldg(X + jj * d + i0 + lane) : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < 32; ++u) xt[lane][warp + NW * u] = ld[u];
        if (tid < 32) xs[tid] = i0 + tid < d ? __ldg(X + row * d + i0 + tid) : 0.0f;
        __syncthreads();
        const int m = min(32, d - i0);
        for (int t = 0; t < m; ++t) {
          const float df = __fsub_rn(xs[t], xt[t][tid]);
          acc = __fadd_rn(acc, __fmul_rn(df, df));
        }
      }
      if (j < j_end && j != row) {
        const uint64_t key = dist_key(__fsqrt_rn(acc), (uint32_t)j);
        if (key < mx) {
          lst[ms * EX_THREADS + tid] = key;
          mx = lst[tid];
          ms = 0;
          for (int t = 1; t < k; ++t) {
            const uint64_t e = lst[t * EX_THREADS + tid];
            if (e > mx) {
              mx = e;
              ms = t;
            }
          }
        }
      }
    }
    __syncthreads();
    for (int p = 0; p < k; ++p) {
      uint64_t mn = ~0ull;
      int sm = 0;
      for (int t = 0; t < k; ++t) {
        const uint64_t e = lst[t * EX_THREADS + tid];
        if (e < mn) {
          mn = e;
          sm = t;
        }
      }
      uint64_t wm = mn;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const uint64_t other = __shfl_xor_sync(0xFFFFFFFFu, wm, o);
        wm = other < wm ? other : wm;
      }
      if (lane == 0) red[warp] = wm;
      __syncthreads();
      uint64_t bm = red[0];
      for (int w = 1; w < EX_THREADS / 32; ++w) bm = red[w] < bm ? red[w] : bm;
      if (bm != ~0ull && mn == bm) lst[sm * EX_THREADS + tid] = ~0ull;
      if (tid == 0) part[((int64_t)b * n_ranges + s) * k + p] = bm;
      __syncthreads();
    }
  }
}

// A warp per listed row: the k smallest of its ranges' keys -> the output row.
__global__ void knn_exact_merge_kernel(const uint64_t* __restrict__ part, const uint32_t* __restrict__ rows,
                                       unsigned n_rows, int n_ranges, int k, uint32_t* __restrict__ out_idx,
                                       float* __restrict__ out_d) {
  const int lane = threadIdx.x & 31;
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= n_rows) return;
  const uint64_t* p = part + w * (int64_t)n_ranges * k;
  const int m = n_ranges * k;
  const int64_t row = rows[w];
  uint64_t prev = 0;
  bool first = true;
  for (int q = 0; q < k; ++q) {
    // smallest key above the previous one (keys are distinct)
    uint64_t mn = ~0ull;
    for (int t = lane; t < m; t += 32) {
      const uint64_t e = p[t];
      if ((first || e > prev) && e < mn) mn = e;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const uint64_t other = __shfl_xor_sync(0xFFFFFFFFu, mn, o);
      mn = other < mn ? other : mn;
    }
    if (lane == 0) {
      out_idx[row * k + q] = mn == ~0ull ? 0u : (uint32_t)mn;
      out_d[row * k + q] = mn == ~0ull ? 0.0f : __uint_as_float((uint32_t)(mn >> 32));
    }
    prev = mn;
    first = false;
    if (mn == ~0ull) {
      for (int r = q + 1 + lane; r < k; r += 32) {
        out_idx[row * k + r] = 0u;
        out_d[row * k + r] = 0.0f;
      }
      break;
    }
  }
}

// Position p of the scan order takes the rank of the locality order (or of the caller's order, perm null) that
// deals each run of 2 S consecutive ranks over the 2 S lists of a group of S tiles, one to a list: a row's
// neighbours, which are near in rank, spread evenly over its lists.  Every run is dealt from another list on
// (a hash of the run), or ranks at a distance of 2 S would all meet in one list: 8,000 rows in 16
// alternating classes, k = 100, had every row recomputed, 21.2 ms against 3.9 for the same rows shuffled.
// Groups are S whole tiles, then one of the whole tiles left; rows past them keep their rank.
__global__ void deal_ranks_kernel(const uint32_t* __restrict__ perm, int64_t n, int S, uint32_t* __restrict__ out) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const int64_t whole = n / DBN, g = p / DBN / S;  // whole tiles, this position's group
  const uint32_t lists = 2u * (uint32_t)min((int64_t)S, whole - g * S);
  int64_t rank = p;
  if (p < whole * DBN) {
    const int64_t first = g * S * DBN;
    const uint32_t at = (uint32_t)(p - first), run = at % (DBN / 2), list = at / (DBN / 2);
    uint32_t h = ((uint32_t)g * (DBN / 2) + run) * 0x9E3779B1u;
    h = (h ^ (h >> 16)) * 0x85EBCA6Bu;
    rank = first + run * lists + (list + ((h >> 16) & 0xFFu)) % lists;
  }
  out[p] = perm ? perm[rank] : (uint32_t)rank;
}

inline unsigned blocks_for(int64_t n, unsigned bt) { return (unsigned)std::min<int64_t>((n + bt - 1) / bt, 1 << 20); }

__global__ void iota_kernel(uint32_t* __restrict__ v, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = (uint32_t)i;
}

// K-d for the listed rows: enough CTAs to fill the GPU (each row's columns split into ranges
// of >= 1024), then the merge.  Synchronises `s`.
void exact_rows(const float* X, int64_t n, int d, int k, const uint32_t* rows, unsigned n_rows, uint32_t* out_idx,
                float* out_dist, cudaStream_t s) {
  const int64_t want = std::max<int64_t>(1, (4 * 148 + (int64_t)n_rows - 1) / (int64_t)n_rows);
  const int ranges = (int)std::max<int64_t>(1, std::min<int64_t>({want, n / 1024 + 1, 256}));
  const unsigned gx = std::min<unsigned>(n_rows, 65535u);
  DevBuf<uint64_t> part((uint64_t)n_rows * ranges * k, s);
  if (k <= KNN_MAX_K)
    knn_exact_part_kernel<256><<<dim3(gx, (unsigned)ranges), 256, (size_t)k * 256 * 8, s>>>(X, n, d, k, rows, n_rows,
                                                                                            ranges, part.p);
  else
    knn_exact_part_kernel<128><<<dim3(gx, (unsigned)ranges), 128, (size_t)k * 128 * 8, s>>>(X, n, d, k, rows, n_rows,
                                                                                            ranges, part.p);
  UB_LAUNCH_CHECK();
  knn_exact_merge_kernel<<<blocks_for((int64_t)n_rows * 32, 256), 256, 0, s>>>(part.p, rows, n_rows, ranges, k,
                                                                               out_idx, out_dist);
  UB_LAUNCH_CHECK();
  UB_CUDA(cudaStreamSynchronize(s));
}

// Database splits of the candidate pass (0: the exact path).  Every (query block, split) pair is one
// work item of a persistent CTA, and every split keeps NCAND candidates per row in two lists of HC.
//  * k <= KNN_MAX_K: halvings of the database until every SM has an item, or 2 tiles are left; three splits
//    instead of two where they take no more waves of items (10,000 x 32, k = 15: 0.62 ms with two, 0.56 with
//    three; with one, whose items are longer but fill one wave, 0.55).  No fewer: a row whose error margin holds
//    more points than its lists (clusters far apart in many dimensions) fails its certificate and is computed
//    again, 20.5 ms for 10,000 x 256 in 50 clusters with one split, 8,587 rows, against 1.0 with three.  And no
//    more: every candidate within the margin is one more exact distance (5,000 x 784 in 10 clusters, k = 10: 1.5
//    ms with four, 2.1 with six).
//  * Longer lists: a row's neighbours fall evenly on the splits' lists (deal_ranks_kernel), each of which
//    keeps HC = 32: 4 splits up to k = 64, else 8, for at most 8 of the k on average (the points within
//    the error margin of the k-th come on top).  A row whose list overflows fails its certificate and
//    is recomputed exactly.
//  * Fewer than LONG_LIST_MIN points and k > KNN_MAX_K: the exact path, which the interface states
//    (rows_recomputed = n; 1,500 x 40, k = 100: 2.3 ms, 2,500 points through the candidate pass 0.5 ms).
constexpr uint64_t LONG_LIST_MIN = 2048;
int pick_splits(uint64_t n, uint64_t k, int64_t q_blocks, int64_t tiles, int sms) {
  if (k > (uint64_t)KNN_MAX_K) {
    if (n < LONG_LIST_MIN) return 0;
    return k <= 64 ? 4 : 8;
  }
  int S = 1;
  while (S < 8 && q_blocks * S < sms && tiles / (2 * S) >= 2) S *= 2;
  const auto waves = [&](int s) { return (q_blocks * s + sms - 1) / sms; };
  return S == 2 && tiles >= 6 && waves(3) == waves(2) ? 3 : S;
}

// Rows whose candidates a call holds at once (a multiple of QM): 512 bytes a row and split, so that the
// scratch of the longest lists (8 splits) stays below 8 GB at any n.  UMAP_B200_KNN_ROWS sets it.
int64_t candidate_rows(int splits) {
  int64_t rows = ((int64_t)8 << 30) / (splits * (int64_t)(NCAND * 8 + 8));
  if (const char* e = getenv("UMAP_B200_KNN_ROWS")) rows = atoll(e);
  return std::max<int64_t>(1, rows / QM) * QM;
}

template <int E>
void launch_rerank(const float* X, int64_t n, int64_t first, int64_t count, int d, int dp, int k, const uint32_t* ci,
                   const float* cd, const float* tau, const float* rn, const unsigned* rmax, float gamma, float scale,
                   const uint32_t* order, uint32_t* oi, float* od, uint32_t* fr, unsigned* fc, cudaStream_t s) {
  knn_rerank_kernel<E><<<blocks_for(count * 32, RERANK_BT), RERANK_BT, 0, s>>>(
      X, n, first, count, d, dp, k, ci, cd, tau, rn, rmax, gamma, scale, order, oi, od, fr, fc);
  UB_LAUNCH_CHECK();
}

}  // namespace

KnnStats knn_bruteforce(const float* X, uint64_t n, uint64_t d, uint64_t k, uint32_t* out_idx, float* out_dist,
                        cudaStream_t s) {
  KnnStats st{};
  if (k < 1 || k > (uint64_t)KNN_MAX_K_EXACT)
    throw Error(INVALID_ARGUMENT, "k must be in 1.." + std::to_string(KNN_MAX_K_EXACT) + ", got " + std::to_string(k));
  if (d < 1 || d > 65536) throw Error(INVALID_ARGUMENT, "dimension must be in 1..65536");
  if (n >= 0x7FFFFF00ull) throw Error(UNSUPPORTED, "n must be < 2^31 - 256");
  if (n == 0) return st;
  if (n == 1) {
    UB_CUDA(cudaMemsetAsync(out_idx, 0, k * 4, s));
    UB_CUDA(cudaMemsetAsync(out_dist, 0, k * 4, s));
    UB_CUDA(cudaStreamSynchronize(s));
    return st;
  }
  {
    // kernel attributes belong to the device's context: set them once per device
    static std::mutex mu;
    static uint64_t done = 0;  // bit per device id < 64
    int dev = 0;
    UB_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if (dev >= 64 || !((done >> dev) & 1u)) {
      UB_CUDA(cudaFuncSetAttribute(knn_candidates_kernel<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)KNN_SMEM));
      UB_CUDA(cudaFuncSetAttribute(knn_candidates_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)KNN_SMEM));
      UB_CUDA(cudaFuncSetAttribute(knn_candidates_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)KNN_SMEM));
      UB_CUDA(cudaFuncSetAttribute(knn_exact_part_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)(KNN_MAX_K * 256 * 8)));
      UB_CUDA(cudaFuncSetAttribute(knn_exact_part_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)(KNN_MAX_K_EXACT * 128 * 8)));
      if (dev < 64) done |= 1ull << dev;
    }
  }
  const int di = (int)d;
  const int64_t dp = (int64_t)((d + KC - 1) / KC) * KC;
  const int64_t n_pad = (int64_t)((n + DBN - 1) / DBN) * DBN;
  const int64_t q_blocks = n_pad / QM, tiles = n_pad / DBN;
  int cur = 0, sms = 148;
  UB_CUDA(cudaGetDevice(&cur));
  UB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, cur));
  const int S = pick_splits(n, k, q_blocks, tiles, sms);
  st.splits = (uint32_t)S;

  DevBuf<double> sums(d, s);
  DevBuf<float> mean(d, s);
  DevBuf<unsigned> flags(5, s);  // 0 non-finite input, 1 max norm, 2 kernel error, 3 failed rows, 4 max |x~|
  UB_CUDA(cudaMemsetAsync(sums.p, 0, d * 8, s));
  UB_CUDA(cudaMemsetAsync(flags.p, 0, 20, s));
  {
    const unsigned gy = (unsigned)std::min<int64_t>(1024, std::max<int64_t>(1, (int64_t)n / 256));
    DevBuf<unsigned> cmm(2 * d, s);
    UB_CUDA(cudaMemsetAsync(cmm.p, 0xFF, d * 4, s));  // min of ordered images starts at the top
    UB_CUDA(cudaMemsetAsync(cmm.p + d, 0, d * 4, s));
    col_sums_kernel<<<dim3((unsigned)((d + 31) / 32), gy), dim3(32, 8), 0, s>>>(X, (int64_t)n, di, sums.p, cmm.p,
                                                                               cmm.p + d, flags.p);
    UB_LAUNCH_CHECK();
    col_means_kernel<<<(unsigned)((d + 255) / 256), 256, 0, s>>>(sums.p, cmm.p, cmm.p + d, (int64_t)n, di, mean.p,
                                                                 flags.p + 4);
    UB_LAUNCH_CHECK();
  }
  unsigned pre[5] = {0, 0, 0, 0, 0};
  UB_CUDA(cudaMemcpyAsync(pre, flags.p, 20, cudaMemcpyDeviceToHost, s));
  UB_CUDA(cudaStreamSynchronize(s));
  if (pre[0]) throw Error(INVALID_ARGUMENT, "kNN input contains NaN or infinite values");
  if (S == 0) {  // every row on the exact CUDA-core path
    DevBuf<uint32_t> all(n, s);
    iota_kernel<<<blocks_for((int64_t)n, 256), 256, 0, s>>>(all.p, (int64_t)n);
    UB_LAUNCH_CHECK();
    exact_rows(X, (int64_t)n, (int)d, (int)k, all.p, (unsigned)n, out_idx, out_dist, s);
    st.fallback_rows = (uint32_t)n;
    st.all_exact = 1;
    return st;
  }
  // scale = 2^e with max |x~| * scale <= 2^14, so every scaled value is finite in FP16
  float maxabs;
  std::memcpy(&maxabs, &pre[4], 4);
  float scale = 1.0f;
  if (maxabs > 0.0f) {
    int e = 0;
    std::frexp(16384.0f / maxabs, &e);
    scale = std::ldexp(1.0f, std::max(-120, std::min(120, e - 1)));
  }
  st.scale = scale;

  DevBuf<__half> xh((uint64_t)(n_pad * dp), s);
  DevBuf<float> nb(n_pad, s), rn(n_pad, s);
  DevBuf<uint32_t> perm;
  const unsigned prep_grid = blocks_for(n_pad * 32, 256);
  if (n >= KNN_REORDER_MIN) {
    // locality order: nearest of NPIV pivot rows (tensor-core GEMM in row chunks), rows
    // sorted by pivot (stable) -> perm[r] = the original row at position r
    DevBuf<__nv_bfloat16> xb((uint64_t)(n_pad * dp), s), piv((uint64_t)NPIV * dp, s);
    DevBuf<float> pn(NPIV, s);
    knn_prep_kernel<<<prep_grid, 256, 0, s>>>(X, (int64_t)n, di, (int)dp, n_pad, mean.p, scale, nullptr, nullptr,
                                              nullptr, xb.p, rn.p, flags.p + 1);
    UB_LAUNCH_CHECK();
    gather_pivots_kernel<<<NPIV, 128, 0, s>>>(xb.p, (int64_t)n, (int)dp, piv.p, pn.p);
    UB_LAUNCH_CHECK();
    constexpr int64_t CH = 65536;
    DevBuf<float> dots((uint64_t)CH * NPIV, s);
    DevBuf<uint32_t> key(n, s), key_sorted(n, s);
    for (int64_t r0 = 0; r0 < (int64_t)n; r0 += CH) {
      const int64_t rows = std::min<int64_t>(CH, n_pad - r0);
      umma_gemm_f32(xb.p + r0 * dp, piv.p, dots.p, rows, NPIV, dp, 1, s);
      nearest_pivot_kernel<<<blocks_for(rows * 32, 256), 256, 0, s>>>(dots.p, rows, r0, (int64_t)n, pn.p, key.p);
      UB_LAUNCH_CHECK();
    }
    DevBuf<uint32_t> sorted(n, s);
    radix_sort_pairs(key.p, nullptr, key_sorted.p, sorted.p, n, 8, s);
    perm.alloc(n, s);
    deal_ranks_kernel<<<blocks_for((int64_t)n, 256), 256, 0, s>>>(sorted.p, (int64_t)n, S, perm.p);
    UB_LAUNCH_CHECK();
    st.reordered = 1;
  } else if (k > (uint64_t)KNN_MAX_K) {
    perm.alloc(n, s);
    deal_ranks_kernel<<<blocks_for((int64_t)n, 256), 256, 0, s>>>(nullptr, (int64_t)n, S, perm.p);
    UB_LAUNCH_CHECK();
  }
  knn_prep_kernel<<<prep_grid, 256, 0, s>>>(X, (int64_t)n, di, (int)dp, n_pad, mean.p, scale, perm.p, xh.p, nb.p, nullptr,
                                            n >= KNN_REORDER_MIN ? nullptr : rn.p, flags.p + 1);
  UB_LAUNCH_CHECK();

  const int64_t q_step = std::min<int64_t>(q_blocks, candidate_rows(S) / QM);
  const uint64_t held = std::min<uint64_t>(n, (uint64_t)q_step * QM);
  const float gamma = (float)(dp + 8) * 9.5367432e-7f;  // (Dp + 8) 2^-20
  DevBuf<uint32_t> cidx(held * S * NCAND, s), fail_rows(n, s);
  DevBuf<uint32_t> lidx((uint64_t)std::min<int64_t>(q_step * S, sms) * 2 * CAP * QM, s);
  DevBuf<float> cdist(held * S * NCAND, s), tau(held * S * 2, s);
  const CUtensorMap tq = bf16_tile_map(xh.p, n_pad, dp, dp, QM, true);
  const CUtensorMap tdb = bf16_tile_map(xh.p, n_pad, dp, dp, DBN, true);
  auto candidates = k <= 16                    ? knn_candidates_kernel<8>
                    : k <= (uint64_t)KNN_MAX_K ? knn_candidates_kernel<16>
                                               : knn_candidates_kernel<0>;
  const int ki = (int)k, dpi = (int)dp;
  cudaEvent_t ev[2];
  UB_CUDA(cudaEventCreate(&ev[0]));
  UB_CUDA(cudaEventCreate(&ev[1]));
  for (int64_t q0 = 0; q0 < q_blocks; q0 += q_step) {
    const int64_t first = q0 * QM, qn = std::min(q_step, q_blocks - q0), count = std::min((int64_t)n - first, qn * QM);
    if (count <= 0) break;  // a last block of padding rows
    UB_CUDA(cudaEventRecord(ev[0], s));
    candidates<<<(unsigned)std::min<int64_t>(qn * S, sms), KNN_THREADS, KNN_SMEM, s>>>(
        tq, tdb, nb.p, (int64_t)n, (int)(dp / KC), tiles, q0, qn, S, ki, di, flags.p + 1, gamma, scale, perm.p, lidx.p,
        cidx.p, cdist.p, tau.p, flags.p + 2);
    UB_LAUNCH_CHECK();
    UB_CUDA(cudaEventRecord(ev[1], s));
    unsigned kerr = 0;
    UB_CUDA(cudaMemcpyAsync(&kerr, flags.p + 2, 4, cudaMemcpyDeviceToHost, s));
    UB_CUDA(cudaStreamSynchronize(s));
    float ms = 0.0f;
    (void)cudaEventElapsedTime(&ms, ev[0], ev[1]);
    st.candidate_ms += ms;
    if (kerr) throw Error(CUDA, "kNN candidate pass: a pipeline wait timed out");
    auto rerank = [&](auto launch) {
      launch(X, (int64_t)n, first, count, di, dpi, ki, cidx.p, cdist.p, tau.p, rn.p, flags.p + 1, gamma, scale, perm.p,
             out_idx, out_dist, fail_rows.p, flags.p + 3, s);
    };
    switch (S) {
      case 1: rerank(launch_rerank<2>); break;
      case 2: rerank(launch_rerank<4>); break;
      case 3: rerank(launch_rerank<6>); break;
      case 4: rerank(launch_rerank<8>); break;
      case 6: rerank(launch_rerank<12>); break;
      default: rerank(launch_rerank<16>); break;
    }
  }
  (void)cudaEventDestroy(ev[0]);
  (void)cudaEventDestroy(ev[1]);
  unsigned n_fail = 0;
  UB_CUDA(cudaMemcpyAsync(&n_fail, flags.p + 3, 4, cudaMemcpyDeviceToHost, s));
  UB_CUDA(cudaStreamSynchronize(s));
  st.fallback_rows = n_fail;
  if (n_fail) exact_rows(X, (int64_t)n, di, ki, fail_rows.p, n_fail, out_idx, out_dist, s);
  return st;
}

}  // namespace ub
