// k nearest neighbours without the N x M distance matrix, three ways (the choice is at the bottom):
//   * many queries, few pairs: one thread per query and a sorted top-k list in registers; reference
//     points stream through shared memory in tiles that every thread of the block reads as a broadcast;
//   * few queries: one or several warps per query, merged at the end;
//   * many pairs, D <= 3: references and queries sorted along a Morton curve, 32 references to a leaf
//     with its bounding box, and a warp per query that only looks at leaves whose box can still hold
//     one of the k nearest points.
// Semantics restated from the reference's include/util/cuda/knn.cuh:
//   distance  :82-103   ssd over the dimensions in order, here pinned to s = fmaf(t, t, s) with
//                       t = ref_i - query_i starting from s = 0
//   selection :125-189  stable insertion, strict '<'  ==  order by (distance, index)
//   indices   :141,160,184  1-based
//   sqrt      :199-205
#include <cub/device/device_radix_sort.cuh>

#include "common.cuh"

namespace mc {

template <int KMAX>
struct TopK {
  float d[KMAX];
  int i[KMAX];
  __device__ __forceinline__ void init() {
#pragma unroll
    for (int t = 0; t < KMAX; ++t) { d[t] = INFINITY; i[t] = -1; }
  }
  __device__ __forceinline__ void insert(float v, int j) {
    d[KMAX - 1] = v;
    i[KMAX - 1] = j;
#pragma unroll
    for (int t = KMAX - 1; t > 0; --t) {
      const bool sw = d[t] < d[t - 1];
      const float dt = d[t], dp = d[t - 1];
      const int it = i[t], ip = i[t - 1];
      d[t] = sw ? dp : dt; d[t - 1] = sw ? dt : dp;
      i[t] = sw ? ip : it; i[t - 1] = sw ? it : ip;
    }
  }
};

// The k <= 32 best of ONE query, spread over a warp: lane t holds the t-th best, ordered by (distance,
// index).  Empty slots are (infinity, 0): nothing at an infinite distance (or NaN) ever enters, as in
// TopK, and such a slot is written as index 0 (= -1 + 1).  A candidate costs about twenty instructions of
// the whole warp and no branch that depends on the lane; a list per lane costs ten times that and is
// walked by the lanes at different times.
struct WarpTopK {
  float d;    // this lane's entry
  int i;
  float thr;  // distance of entry k - 1: candidates beyond it cannot enter (warp uniform)

  static __device__ __forceinline__ bool less(float da, int ia, float db, int ib) {
    return da < db || (da == db && ia < ib);
  }
  __device__ __forceinline__ void init() { d = INFINITY; i = 0; thr = INFINITY; }
  // first 32 candidates, one per lane: sorted at once
  __device__ __forceinline__ void fill(float s, int j, int k, int lane) {
    const bool ok = s < INFINITY;
    d = ok ? s : INFINITY;
    i = ok ? j : 0;
#pragma unroll
    for (int size = 2; size <= 32; size *= 2) {
#pragma unroll
      for (int o = size / 2; o > 0; o /= 2) {
        const float od = __shfl_xor_sync(0xffffffffu, d, o);
        const int oi = __shfl_xor_sync(0xffffffffu, i, o);
        const bool low = ((lane & o) == 0) == ((lane & size) == 0);  // this lane keeps the smaller one
        if (less(od, oi, d, i) == low) { d = od; i = oi; }
      }
    }
    thr = __shfl_sync(0xffffffffu, d, k - 1);
  }
  // one candidate per lane; those within thr enter one after another.  IN_ORDER: candidates come in index
  // order, so that one at distance thr cannot displace anything.
  template <bool IN_ORDER>
  __device__ __forceinline__ void offer(float s, int j, int k, int lane) {
    unsigned m = __ballot_sync(0xffffffffu, IN_ORDER ? s < thr : s <= thr && s < INFINITY);
    while (m) {
      const int src = __ffs(m) - 1;
      m &= m - 1;
      const float cs = __shfl_sync(0xffffffffu, s, src);
      const int cj = __shfl_sync(0xffffffffu, j, src);
      if (IN_ORDER ? cs >= thr : cs > thr) continue;
      const float ud = __shfl_up_sync(0xffffffffu, d, 1);
      const int ui = __shfl_up_sync(0xffffffffu, i, 1);
      if (less(cs, cj, d, i)) {
        const bool above = lane > 0 && less(cs, cj, ud, ui);
        d = above ? ud : cs;
        i = above ? ui : cj;
      }
      thr = __shfl_sync(0xffffffffu, d, k - 1);
    }
  }
};

// The queries of an all-pairs kernel.  On its own it takes all of them.  Behind the search among sorted leaves it
// takes what the search has left: everything where the references are crowded (see knn_leaves_kernel), else the
// queries that were listed (see knn_tree_kernel) - a warp or several per query where these are few.
struct KnnTodo {
  const int* crowded;  // leaves in crowded places; null: not behind a search
  const int* count;    // [B] queries listed
  const int* list;     // [B][N]
  int nleaf;           // leaves in all
  int few;             // up to here: warps per query
  __device__ __forceinline__ bool searched() const { return __ldg(crowded) <= nleaf / 8; }
  // how many queries of batch b there are, and their list (null: 0, 1, ..)
  __device__ __forceinline__ int take(int b, int N, const int** from) const {
    *from = nullptr;
    if (!crowded || !searched()) return N;
    *from = list + (long)b * N;
    return __ldg(count + b);
  }
};

constexpr int KNN_THREADS = 256;
constexpr int KNN_TILE = 512;
constexpr int KNN_DMAX = 16;
constexpr int KNNT_DMAX = 3;  // dimensions the search among sorted leaves takes

// ---- few queries: a warp, or several, per query -----------------------------------------------------
// One thread per query leaves the chip idle when there are few: 200 queries are two blocks of the kernels
// below, whose threads walk 160 000 references one after another (2.9 ms).  Here the lanes of a warp look
// at 32 references at a time (coalesced loads, four in flight per coordinate) for one query, whose list is
// spread over the lanes; wpq warps share a query's references and the first one merges their lists.
constexpr int KNNW_WARPS = 8;       // warps of a block that takes several queries
constexpr int KNNW_MAX_WARPS = 32;  // warps that share one query at most

// Enough warps for the chip, at least 16 references per lane.
__host__ __device__ __forceinline__ int knn_warps_per_query(long queries, int M, int most) {
  int wpq = 1;
  while (wpq < most && queries * wpq < 148 * 16 && M >= 2 * wpq * 32 * 16) wpq *= 2;
  return wpq;
}

__device__ __forceinline__ void knn_store(int64_t* idx, float* dist, long o, float d, int i) {
  idx[o] = d == INFINITY ? 0 : (int64_t)i + 1;
  dist[o] = __fsqrt_rn(d);
}

// Queries [0, total) of batch b (through `from`, if any), dealt out to the grid's blocks; sd, si: one row per warp.
template <int DT>
__device__ __forceinline__ void knn_wide(const float* __restrict__ ref, const float* __restrict__ query, int D, int M,
                                         int N, int k, int64_t* __restrict__ idx, float* __restrict__ dist, int b,
                                         const int* from, int total, float (*sd)[32], int (*si)[32]) {
  constexpr int DS = DT > 0 ? DT : KNN_DMAX;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int warps = blockDim.x >> 5, wpq = knn_warps_per_query((long)total * gridDim.y, M, warps), qpb = warps / wpq;
  const int part = warp % wpq;
  const float* rb = ref + (long)b * D * M;
  const float* qb = query + (long)b * D * N;
  for (int q0 = blockIdx.x * qpb; q0 < total; q0 += gridDim.x * qpb) {
    const int slot = q0 + warp / wpq;
    const bool live = slot < total;
    const int n = live && from ? __ldg(from + slot) : slot;
    WarpTopK top;
    top.init();
    if (live) {
      float q[DS];
#pragma unroll
      for (int i = 0; i < DS; ++i) q[i] = i < D ? __ldg(qb + (long)i * N + n) : 0.f;
      constexpr int U = 4;
      bool first = true;
      for (int m0 = part * 32; m0 < M; m0 += wpq * 32 * U) {
        float s[U];
#pragma unroll
        for (int u = 0; u < U; ++u) s[u] = 0.f;
#pragma unroll
        for (int i = 0; i < DS; ++i) {
          if (DT == 0 && i >= D) break;
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int j = m0 + u * wpq * 32 + lane;
            const float t = (j < M ? __ldg(rb + (long)i * M + j) : INFINITY) - q[i];
            s[u] = fmaf(t, t, s[u]);
          }
        }
        int u0 = 0;
        if (first) { top.fill(s[0], m0 + lane, k, lane); first = false; u0 = 1; }
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (u >= u0) top.offer<true>(s[u], m0 + u * wpq * 32 + lane, k, lane);
      }
    }
    if (wpq > 1) {
      sd[warp][lane] = top.d;
      si[warp][lane] = top.i;
      __syncthreads();
      if (part == 0)
        for (int p = 1; p < wpq; ++p)
          top.offer<false>(lane < k ? sd[warp + p][lane] : INFINITY, si[warp + p][lane], k, lane);
      __syncthreads();
    }
    if (part == 0 && live && lane < k) knn_store(idx, dist, ((long)b * k + lane) * N + n, top.d, top.i);
  }
}

template <int DT>
__global__ void __launch_bounds__(KNNW_MAX_WARPS * 32, 1) knn_wide_kernel(const float* __restrict__ ref,
                                                                      const float* __restrict__ query, int D, int M,
                                                                      int N, int k, int64_t* __restrict__ idx,
                                                                      float* __restrict__ dist) {
  __shared__ float sd[KNNW_MAX_WARPS][32];
  __shared__ int si[KNNW_MAX_WARPS][32];
  knn_wide<DT>(ref, query, D, M, N, k, idx, dist, blockIdx.y, nullptr, N, sd, si);
}

// ---- one thread per query ---------------------------------------------------------------------------
// DT > 0: compile-time dimension; DT == 0: runtime dimension up to KNN_DMAX.
template <int DT, int KMAX>
__global__ void __launch_bounds__(KNN_THREADS) knn_kernel(const float* __restrict__ ref,
                                                          const float* __restrict__ query, int D,
                                                          int M, int N, int k,
                                                          int64_t* __restrict__ idx,
                                                          float* __restrict__ dist, KnnTodo todo) {
  constexpr int DS = DT > 0 ? DT : KNN_DMAX;
  __shared__ float tile[DS][KNN_TILE];
  const int b = blockIdx.y;
  const float* rb = ref + (long)b * D * M;
  const float* qb = query + (long)b * D * N;
  const int* from;
  const int total = todo.take(b, N, &from);
  if constexpr (DT > 0 && DT <= KNNT_DMAX) {
    if (todo.crowded && total <= todo.few) {
      __shared__ float sd[KNN_THREADS / 32][32];
      __shared__ int si[KNN_THREADS / 32][32];
      knn_wide<DT>(ref, query, D, M, N, k, idx, dist, b, from, total, sd, si);
      return;
    }
  }
  if (blockIdx.x * KNN_THREADS >= (unsigned)total) return;
  const int slot = blockIdx.x * KNN_THREADS + threadIdx.x;
  const bool live = slot < total;
  const int n = live && from ? __ldg(from + slot) : slot;
  float q[DS];
#pragma unroll
  for (int i = 0; i < DS; ++i) q[i] = (live && i < D) ? qb[(long)i * N + n] : 0.f;
  TopK<KMAX> top;
  top.init();

  for (int m0 = 0; m0 < M; m0 += KNN_TILE) {
    const int cnt = min(KNN_TILE, M - m0);
    __syncthreads();
    for (int t = threadIdx.x; t < DS * KNN_TILE; t += KNN_THREADS) {
      const int i = t / KNN_TILE, j = t % KNN_TILE;
      tile[i][j] = (i < D && j < cnt) ? rb[(long)i * M + m0 + j] : 0.f;
    }
    __syncthreads();
    if (live) {
#pragma unroll 4
      for (int j = 0; j < cnt; ++j) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < DS; ++i) {
          const float t = tile[i][j] - q[i];
          s = fmaf(t, t, s);
        }
        if (s < top.d[KMAX - 1]) top.insert(s, m0 + j);
      }
    }
  }
  if (!live) return;
#pragma unroll
  for (int t = 0; t < KMAX; ++t) {
    if (t < k) {
      const long o = ((long)b * k + t) * N + n;
      idx[o] = (int64_t)top.i[t] + 1;
      dist[o] = __fsqrt_rn(top.d[t]);
    }
  }
}

// D <= 4: reference points are staged per coordinate and visited two at a time with packed
// fp32 arithmetic (fma.rn.f32x2): difference and square-accumulate of a PAIR of references cost
// one instruction each per dimension.  Every lane of a packed operation is the same correctly
// rounded operation as its scalar form (r - q as fma(r, 1, -q), then s = fma(t, t, s) from 0), so
// distances - and with them the order of near ties - are bit-identical to the scalar kernel.
// Blocks of 128 threads, nine to an SM (56 registers): 170 496 resident queries, so that the
// 163 842 vertices of a level-7 icosphere run as ONE wave instead of one full wave and a sliver.
constexpr int KNN2_THREADS = 128;
constexpr int KNN2_BLOCKS_PER_SM = 9;
constexpr int KNN2_TILE = 1024;

__device__ __forceinline__ float2 fma2(const float2& a, const float2& b, const float2& c) {
  float2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<const unsigned long long&>(a)),
        "l"(reinterpret_cast<const unsigned long long&>(b)),
        "l"(reinterpret_cast<const unsigned long long&>(c)));
  return d;
}

template <int DT, int KMAX>
__global__ void __launch_bounds__(KNN2_THREADS, KMAX <= 12 ? KNN2_BLOCKS_PER_SM : 8) knn_small_d_kernel(const float* __restrict__ ref,
                                                                   const float* __restrict__ query,
                                                                   int M, int N, int k,
                                                                   int64_t* __restrict__ idx,
                                                                   float* __restrict__ dist, KnnTodo todo) {
  __shared__ __align__(16) float tile[DT][KNN2_TILE];
  const int b = blockIdx.y;
  const float* rb = ref + (long)b * DT * M;
  const float* qb = query + (long)b * DT * N;
  const int* from;
  const int total = todo.take(b, N, &from);
  if constexpr (DT > 0 && DT <= KNNT_DMAX) {
    if (todo.crowded && total <= todo.few) {
      __shared__ float sd[KNN2_THREADS / 32][32];
      __shared__ int si[KNN2_THREADS / 32][32];
      knn_wide<DT>(ref, query, DT, M, N, k, idx, dist, b, from, total, sd, si);
      return;
    }
  }
  if (blockIdx.x * KNN2_THREADS >= (unsigned)total) return;
  const int slot = blockIdx.x * KNN2_THREADS + threadIdx.x;
  const bool live = slot < total;
  const int n = live && from ? __ldg(from + slot) : slot;
  float2 nq[DT];  // (-q_i, -q_i)
#pragma unroll
  for (int i = 0; i < DT; ++i) {
    const float v = live ? qb[(long)i * N + n] : 0.f;
    nq[i] = make_float2(-v, -v);
  }
  const float2 one = make_float2(1.f, 1.f), zero = make_float2(0.f, 0.f);
  TopK<KMAX> top;
  top.init();
  for (int m0 = 0; m0 < M; m0 += KNN2_TILE) {
    const int cnt = min(KNN2_TILE, M - m0);
    const int cnt2 = (cnt + 3) & ~3;  // the tail is padded with points at infinity
    __syncthreads();
    for (int j = threadIdx.x; j < cnt2; j += KNN2_THREADS) {
#pragma unroll
      for (int i = 0; i < DT; ++i) tile[i][j] = j < cnt ? rb[(long)i * M + m0 + j] : INFINITY;
    }
    __syncthreads();
    if (live) {
#pragma unroll 2
      for (int j = 0; j < cnt2; j += 4) {
        float2 s0 = zero, s1 = zero;
#pragma unroll
        for (int i = 0; i < DT; ++i) {
          const float4 r = *reinterpret_cast<const float4*>(&tile[i][j]);
          const float2 t0 = fma2(make_float2(r.x, r.y), one, nq[i]);  // r - q
          const float2 t1 = fma2(make_float2(r.z, r.w), one, nq[i]);
          s0 = fma2(t0, t0, s0);
          s1 = fma2(t1, t1, s1);
        }
        // one test for the four candidates; the list is rarely touched after the first few tiles
        if (fminf(fminf(s0.x, s0.y), fminf(s1.x, s1.y)) < top.d[KMAX - 1]) {
          if (s0.x < top.d[KMAX - 1]) top.insert(s0.x, m0 + j);
          if (s0.y < top.d[KMAX - 1]) top.insert(s0.y, m0 + j + 1);
          if (s1.x < top.d[KMAX - 1]) top.insert(s1.x, m0 + j + 2);
          if (s1.y < top.d[KMAX - 1]) top.insert(s1.y, m0 + j + 3);
        }
      }
    }
  }
  if (!live) return;
#pragma unroll
  for (int t = 0; t < KMAX; ++t) {
    if (t < k) {
      const long o = ((long)b * k + t) * N + n;
      idx[o] = (int64_t)top.i[t] + 1;
      dist[o] = __fsqrt_rn(top.d[t]);
    }
  }
}


// ---- many pairs: leaves on a Morton curve -----------------------------------------------------------
// 163 842 x 163 842 points are 2.7e10 pairs: 7.6 ms at the rate of the packed arithmetic above, while
// all but about a hundred references per query can be ruled out by their position.  Keys of all
// references and queries (segment, 24-bit Morton code inside the bounding box of the references) are
// radix sorted; 32 consecutive references of the order form a leaf, 32 leaves a node, 32 nodes a
// group, each with the bounding box of its points.  A warp takes one query at a time: it starts with the
// leaf where the query stands in the order (sorted at once), then its lanes test 32 boxes at a time and
// the warp visits - one reference per lane - the leaves whose box is not farther from the query than its
// k-th distance so far.  Consecutive warps take consecutive queries of the order, so that they meet the
// same leaves in L1.
// The box distance is formed like the point distance, with the gap to the box in place of the
// coordinate difference: rounding is monotone, so it is never above the computed distance of any point
// in the box, and "skip if box distance > k-th distance" cannot lose a point, ties included (equal
// distances are ordered by index, hence no skip at equality).
// NaN references are outside every box and never nearer than anything.
// What a box rules out depends on the queries too: one in the middle of a sphere of references, or far from all of
// them, is about as far from every leaf and would visit them all, 32 points at a time, at up to four times the
// cost of all pairs.  A query that has visited a quarter of the leaves is therefore given up and listed for the
// all-pairs kernels, and once a thirty-second of a batch's queries is listed, others that have visited 64 leaves
// follow.  163 842 references on the sphere and as many queries at its centre 34.1 -> 9.9 ms (all pairs: 8.4 ms), 160 000
// and 2 000 1.59 -> 1.02 ms; queries on the sphere 312 -> 323 us.
// (Tried first: one query per lane and 32 neighbouring queries per warp, every lane testing the points of
// all leaves that one of them needs: 271 us for the search alone, and far slower than all pairs where
// queries are sparse among the references.)
constexpr int KNNT_LEAF = 32;
constexpr int KNNT_WARPS = 4;
constexpr int KNNT_BITS = 24;

__device__ __forceinline__ unsigned float_order(float f) {  // unsigned order == float order
  const unsigned u = __float_as_uint(f);
  return (u >> 31) ? ~u : u | 0x80000000u;
}
__device__ __forceinline__ float float_unorder(unsigned u) {
  return __uint_as_float((u >> 31) ? u & 0x7fffffffu : ~u);
}

// bounds[b][0][i] = max of ~order(x) (i.e. the minimum), bounds[b][1][i] = max of order(x); zeroed before
template <int DT>
__global__ void __launch_bounds__(256) knn_bounds_kernel(const float* __restrict__ ref, int M,
                                                         unsigned* __restrict__ bounds) {
  const int b = blockIdx.y;
  unsigned lo[DT], hi[DT];
#pragma unroll
  for (int i = 0; i < DT; ++i) lo[i] = hi[i] = 0u;
  for (int j = blockIdx.x * 256 + threadIdx.x; j < M; j += gridDim.x * 256) {
#pragma unroll
    for (int i = 0; i < DT; ++i) {
      const float v = __ldg(ref + ((long)b * DT + i) * M + j);
      if (fabsf(v) <= FLT_MAX) {  // (no NaN, no infinity)
        const unsigned o = float_order(v);
        lo[i] = max(lo[i], ~o);
        hi[i] = max(hi[i], o);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < DT; ++i) {
    lo[i] = __reduce_max_sync(0xffffffffu, lo[i]);
    hi[i] = __reduce_max_sync(0xffffffffu, hi[i]);
    if ((threadIdx.x & 31) == 0) {
      atomicMax(bounds + ((long)b * 2 + 0) * DT + i, lo[i]);
      atomicMax(bounds + ((long)b * 2 + 1) * DT + i, hi[i]);
    }
  }
}

template <int DT>
__device__ __forceinline__ unsigned morton_spread(unsigned v) {
  if (DT == 1) return v;
  if (DT == 2) {
    v = (v | (v << 8)) & 0x00FF00FFu; v = (v | (v << 4)) & 0x0F0F0F0Fu;
    v = (v | (v << 2)) & 0x33333333u; return (v | (v << 1)) & 0x55555555u;
  }
  v = (v | (v << 16)) & 0x030000FFu; v = (v | (v << 8)) & 0x0300F00Fu;
  v = (v | (v << 4)) & 0x030C30C3u;
  return (v | (v << 2)) & 0x09249249u;
}

// key = segment << 24 | code; segments 0 .. B-1 are the references, B .. 2 B - 1 the queries
template <int DT>
__global__ void __launch_bounds__(256) knn_keys_kernel(const float* __restrict__ ref,
                                                       const float* __restrict__ query, int B, int M, int N,
                                                       const unsigned* __restrict__ bounds,
                                                       unsigned* __restrict__ keys, int* __restrict__ vals) {
  constexpr int BITS = KNNT_BITS / DT;
  const long nref = (long)B * M, total = nref + (long)B * N;
  for (long t = blockIdx.x * 256L + threadIdx.x; t < total; t += gridDim.x * 256L) {
    const bool isq = t >= nref;
    const long r = isq ? t - nref : t;
    const int n = isq ? N : M;
    const int b = (int)(r / n), j = (int)(r - (long)b * n);
    unsigned code = 0;
#pragma unroll
    for (int i = 0; i < DT; ++i) {
      const float v = __ldg((isq ? query : ref) + ((long)b * DT + i) * n + j);
      const float lo = float_unorder(~__ldg(bounds + ((long)b * 2 + 0) * DT + i));
      const float hi = float_unorder(__ldg(bounds + ((long)b * 2 + 1) * DT + i));
      float f = (v - lo) * ((float)(1 << BITS) / fmaxf(hi - lo, 1e-37f));
      f = fminf(fmaxf(f, 0.f), (float)((1 << BITS) - 1));  // (NaN becomes 0)
      code |= morton_spread<DT>((unsigned)f) << i;
    }
    keys[t] = (unsigned)(isq ? B + b : b) << KNNT_BITS | code;
    vals[t] = j;
  }
}

// Leaf l of batch b: coordinates [DT][32] and original indices [32].  Boxes are stored 32 siblings
// together, component by component - [parent][lo 0 .. lo DT-1, hi 0 .. hi DT-1][32] - so that a warp
// reads each component of 32 boxes in one run (as structs they cost six times the L1 wavefronts, which
// was half of the search's time); missing siblings are empty boxes, at infinite distance.
// One warp per leaf, one block of 32 warps per node.
// A curve of 8 bits per dimension cannot tell the points of one cell apart: a leaf whose cell fills 64
// leaves and more is counted as crowded, and with more than an eighth of such leaves (points that nearly
// all sit in one spot) the all-pairs kernels do the work instead.
template <int DT>
__global__ void __launch_bounds__(1024) knn_leaves_kernel(const float* __restrict__ ref, int M, int nleaf,
                                                          const unsigned* __restrict__ keys,
                                                          const int* __restrict__ vals, float* __restrict__ leaves,
                                                          float* __restrict__ lbox, float* __restrict__ nbox,
                                                          int ngroup, int* __restrict__ crowded) {
  __shared__ float sb[2 * DT][32];
  const int b = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int node = blockIdx.x, l = node * 32 + warp;
  const int p = l * KNNT_LEAF + lane;
  const bool on = l < nleaf && p < M;
  const int j = on ? __ldg(vals + (long)b * M + p) : 0;
  float* lb = lbox + ((long)b * gridDim.x + node) * (2 * DT * 32);
#pragma unroll
  for (int i = 0; i < DT; ++i) {
    const float v = on ? __ldg(ref + ((long)b * DT + i) * M + j) : INFINITY;
    float lo = on ? v : INFINITY, hi = on ? v : -INFINITY;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {  // (fminf / fmaxf leave NaN coordinates out)
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) {
      lb[i * 32 + warp] = sb[i][warp] = lo;
      lb[(DT + i) * 32 + warp] = sb[DT + i][warp] = hi;
    }
    if (l < nleaf) leaves[((long)b * nleaf + l) * ((DT + 1) * KNNT_LEAF) + i * KNNT_LEAF + lane] = v;
  }
  if (l < nleaf)
    reinterpret_cast<int*>(leaves)[((long)b * nleaf + l) * ((DT + 1) * KNNT_LEAF) + DT * KNNT_LEAF + lane] = j;
  if (lane == 0 && l + 64 < nleaf && __ldg(keys + (long)b * M + p) == __ldg(keys + (long)b * M + p + 64 * KNNT_LEAF))
    atomicAdd(crowded, 1);
  __syncthreads();
  if (warp == 0) {
    float* nb = nbox + ((long)b * ngroup + (node >> 5)) * (2 * DT * 32) + (node & 31);
#pragma unroll
    for (int i = 0; i < DT; ++i) {
      float lo = sb[i][lane], hi = sb[DT + i][lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      }
      if (lane == 0) { nb[i * 32] = lo; nb[(DT + i) * 32] = hi; }
    }
  }
}

// Boxes of the groups, one warp per 32 nodes; also empties the slots behind the last node and group.
template <int DT>
__global__ void __launch_bounds__(32) knn_groups_kernel(float* __restrict__ nbox, int nnode, int ngroup,
                                                        float* __restrict__ gbox) {
  const int b = blockIdx.y, lane = threadIdx.x, g = blockIdx.x;
  float* nb = nbox + ((long)b * ngroup + g) * (2 * DT * 32) + lane;  // (not read for g >= ngroup)
  float* gb = gbox + ((long)b * (gridDim.x / 32) + (g >> 5)) * (2 * DT * 32) + (g & 31);
  const bool on = g * 32 + lane < nnode;
#pragma unroll
  for (int i = 0; i < DT; ++i) {
    float lo = on ? nb[i * 32] : INFINITY, hi = on ? nb[(DT + i) * 32] : -INFINITY;
    if (!on && g < ngroup) { nb[i * 32] = INFINITY; nb[(DT + i) * 32] = -INFINITY; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if (lane == 0) { gb[i * 32] = lo; gb[(DT + i) * 32] = hi; }
  }
}

// Squared gap between a point and this lane's box of 32 siblings, formed like a point distance.
template <int DT>
__device__ __forceinline__ float box_gap2(const float (&q)[DT], const float* __restrict__ bx) {
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < DT; ++i) {
    const float t = fmaxf(fmaxf(__ldg(bx + i * 32) - q[i], q[i] - __ldg(bx + (DT + i) * 32)), 0.f);
    s = fmaf(t, t, s);
  }
  return s;
}

// Lane with the smallest gap if that is within thr, else -1; its gap is struck out.
__device__ __forceinline__ int pop_nearest(float& gap, float thr, int lane) {
  const unsigned m = __reduce_min_sync(0xffffffffu, __float_as_uint(gap));  // (gaps are >= 0)
  if (m >= 0x7f800000u || __uint_as_float(m) > thr) return -1;
  const int src = __ffs(__ballot_sync(0xffffffffu, __float_as_uint(gap) == m)) - 1;
  if (lane == src) gap = INFINITY;
  return src;
}

// qkeys: sorted keys of the queries; null: the queries are the references themselves, and a query's place
// in the order is its leaf slot.
template <int DT>
__global__ void __launch_bounds__(KNNT_WARPS * 32) knn_tree_kernel(
    const float* __restrict__ query, int M, int N, int k, int nleaf, int nnode, int ngroup,
    const unsigned* __restrict__ keys, const unsigned* __restrict__ qkeys, const int* __restrict__ qvals,
    const float* __restrict__ leaves, const float* __restrict__ lbox, const float* __restrict__ nbox,
    const float* __restrict__ gbox, KnnTodo todo, int* __restrict__ listed, int* __restrict__ list, int budget,
    int64_t* __restrict__ idx, float* __restrict__ dist) {
  if (!todo.searched()) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int b = blockIdx.y;
  constexpr int LSTRIDE = (DT + 1) * KNNT_LEAF, BSTRIDE = 2 * DT * 32;
  const float* lf = leaves + (long)b * nleaf * LSTRIDE + lane;
  const float* lb = lbox + (long)b * nnode * BSTRIDE + lane;
  const float* nb = nbox + (long)b * ngroup * BSTRIDE + lane;
  const float* gb = gbox + (long)b * ((ngroup + 31) / 32) * BSTRIDE + lane;
  const int pos = blockIdx.x * KNNT_WARPS + warp;
  if (pos >= N) return;
  const int n = __ldg(qvals + (long)b * N + pos);
  float q[DT];
#pragma unroll
  for (int i = 0; i < DT; ++i) q[i] = __ldg(query + ((long)b * DT + i) * N + n);
  // where the query stands among the references: that leaf comes first
  int at = pos / KNNT_LEAF;
  if (qkeys) {
    const unsigned key = (__ldg(qkeys + (long)b * N + pos) & ((1u << KNNT_BITS) - 1)) | (unsigned)b << KNNT_BITS;
    const unsigned* ks = keys + (long)b * M;
    int lo = 0, len = M;  // lower bound, 32 probes at a time
    while (len > 0) {
      const int step = (len + 31) / 32;
      const int p = lane * step;
      const bool below = p < len && __ldg(ks + lo + p) < key;
      const int c = __popc(__ballot_sync(0xffffffffu, below));
      if (c == 0) break;
      lo += (c - 1) * step + 1;
      len = min(step - 1, len - (c - 1) * step - 1);
    }
    at = min(lo, M - 1) / KNNT_LEAF;
  }
  auto point = [&](int l, float& s, int& j) {  // this lane's reference of leaf l
    const float* p = lf + (long)l * LSTRIDE;
    s = 0.f;
#pragma unroll
    for (int i = 0; i < DT; ++i) {
      const float t = __ldg(p + i * KNNT_LEAF) - q[i];
      s = fmaf(t, t, s);
    }
    j = __float_as_int(__ldg(p + DT * KNNT_LEAF));
  };
  WarpTopK top;
  float s;
  int j;
  point(at, s, j);
  top.fill(s, j, k, lane);
  // Nearest box first on every level: a leaf may hold points from both sides of a jump of the curve, so
  // that the first k-th distance is far too large for a few queries, and these would visit thousands
  // of leaves in index order (4 x the time of the whole search).
  // (a NaN coordinate is at no distance from anything: the list stays empty, and no box may be asked -
  // NaN would pass for a gap of zero, in empty slots as well)
  bool nan = false;
#pragma unroll
  for (int i = 0; i < DT; ++i) nan |= q[i] != q[i];
  int seen = 0;  // leaves visited
  for (int g0 = 0; g0 < ngroup && !nan; g0 += 32) {
    float ggap = box_gap2<DT>(q, gb + (g0 / 32) * BSTRIDE);
    for (int gs; (gs = pop_nearest(ggap, top.thr, lane)) >= 0;) {
      const int n0 = (g0 + gs) * 32;
      float ngap = box_gap2<DT>(q, nb + (long)(g0 + gs) * BSTRIDE);
      for (int ns; (ns = pop_nearest(ngap, top.thr, lane)) >= 0;) {
        const int l0 = (n0 + ns) * 32;
        float lgap = box_gap2<DT>(q, lb + (long)(n0 + ns) * BSTRIDE);
        if (l0 + lane == at) lgap = INFINITY;
        for (int ls; (ls = pop_nearest(lgap, top.thr, lane)) >= 0;) {
          point(l0 + ls, s, j);
          top.offer<false>(s, j, k, lane);
        }
        // (added up per node: a counter in the loop over leaves makes the search 8 % slower)
        seen += __popc(__ballot_sync(0xffffffffu, lgap == INFINITY));
        if (seen > 64) {
          int others = lane == 0 ? *(volatile const int*)(listed + b) : 0;
          others = __shfl_sync(0xffffffffu, others, 0);
          if (seen > budget || others > N / 32) top.thr = -1.f;  // (no box passes any more)
        }
      }
    }
  }
  if (top.thr < 0.f) {
    if (lane == 0) list[(long)b * N + atomicAdd(listed + b, 1)] = n;
    return;
  }
  if (lane < k) knn_store(idx, dist, ((long)b * k + lane) * N + n, top.d, top.i);
}

struct KnnTreeWs {
  size_t list, bounds, keys_in, keys, vals_in, vals, leaves, lbox, nbox, gbox, cub, cub_bytes, total;
  long items;
  int nleaf, nnode, ngroup, end_bit;
};

static KnnTreeWs knn_tree_layout(int B, int D, int M, int N, bool same) {
  KnnTreeWs L;
  L.items = (long)B * M + (same ? 0 : (long)B * N);
  L.nleaf = (M + KNNT_LEAF - 1) / KNNT_LEAF;
  L.nnode = (L.nleaf + 31) / 32;
  L.ngroup = (L.nnode + 31) / 32;
  L.end_bit = KNNT_BITS;
  while ((1L << (L.end_bit - KNNT_BITS)) < (same ? B : 2L * B)) ++L.end_bit;
  size_t o = 0;
  auto take = [&](size_t n) { const size_t at = o; o += (n + 255) & ~(size_t)255; return at; };
  L.bounds = take((size_t)B * (2 * D + 1) * 4 + 16);  // (and the counts of listed queries and crowded leaves)
  L.list = take((size_t)B * N * 4);
  L.keys_in = take((size_t)L.items * 4);
  L.keys = take((size_t)L.items * 4);
  L.vals_in = take((size_t)L.items * 4);
  L.vals = take((size_t)L.items * 4);
  L.leaves = take((size_t)B * L.nleaf * (D + 1) * KNNT_LEAF * 4);
  L.lbox = take((size_t)B * L.nnode * 2 * D * 128);
  L.nbox = take((size_t)B * L.ngroup * 2 * D * 128);
  L.gbox = take((size_t)B * ((L.ngroup + 31) / 32) * 2 * D * 128);
  L.cub_bytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, L.cub_bytes, (const unsigned*)nullptr, (unsigned*)nullptr,
                                  (const int*)nullptr, (int*)nullptr, (int)L.items, 0, L.end_bit);
  L.cub = take(L.cub_bytes);
  L.total = o;
  return L;
}

template <int DT>
static void knn_thread_launch(const float* ref, const float* query, int B, int D, int M, int N, int k,
                              int64_t* idx, float* dist, cudaStream_t st, const KnnTodo& todo);
static long knn_few(int D, int M);

template <int DT>
static int knn_tree_launch(const float* ref, const float* query, int B, int M, int N, int k, int64_t* idx,
                           float* dist, void* ws, size_t ws_bytes, cudaStream_t st) {
  const bool same = ref == query && M == N;
  const KnnTreeWs L = knn_tree_layout(B, DT, M, N, same);
  if (!ws || ws_bytes < L.total) return MC_ERR_WORKSPACE;
  if (((uintptr_t)ws) & 15) return MC_ERR_BAD_ARG;
  uint8_t* p = (uint8_t*)ws;
  unsigned *bounds = (unsigned*)(p + L.bounds), *keys_in = (unsigned*)(p + L.keys_in), *keys = (unsigned*)(p + L.keys);
  int *vals_in = (int*)(p + L.vals_in), *vals = (int*)(p + L.vals);
  float *leaves = (float*)(p + L.leaves), *lbox = (float*)(p + L.lbox), *nbox = (float*)(p + L.nbox),
        *gbox = (float*)(p + L.gbox);
  int* listed = (int*)(bounds + (long)B * 2 * DT);
  int* crowded = listed + B;
  int* list = (int*)(p + L.list);
  if (cudaMemsetAsync(bounds, 0, (size_t)B * (2 * DT + 1) * 4 + 4, st) != cudaSuccess) return MC_ERR_LAUNCH;
  int bb = (M + 1023) / 1024;
  if (bb > 148) bb = 148;
  knn_bounds_kernel<DT><<<dim3(bb, B), 256, 0, st>>>(ref, M, bounds), MC_COUNT(1);
  knn_keys_kernel<DT><<<grid_for(L.items, 256), 256, 0, st>>>(ref, query, B, M, same ? 0 : N, bounds, keys_in, vals_in),
      MC_COUNT(1);
  size_t cb = L.cub_bytes;
  if (cub::DeviceRadixSort::SortPairs(p + L.cub, cb, keys_in, keys, vals_in, vals, (int)L.items, 0, L.end_bit, st) !=
      cudaSuccess)
    return MC_ERR_LAUNCH;
  knn_leaves_kernel<DT><<<dim3(L.nnode, B), 1024, 0, st>>>(ref, M, L.nleaf, keys, vals, leaves, lbox, nbox, L.ngroup,
                                                           crowded), MC_COUNT(1);
  knn_groups_kernel<DT><<<dim3((L.ngroup + 31) / 32 * 32, B), 32, 0, st>>>(nbox, L.nnode, L.ngroup, gbox), MC_COUNT(1);
  const KnnTodo todo = {crowded, listed, list, L.nleaf * B, (int)(knn_few(DT, M) / B)};
  const int budget = L.nleaf / 4 > 128 ? L.nleaf / 4 : 128;
  const unsigned* qkeys = same ? nullptr : keys + (long)B * M;
  const int* qvals = same ? vals : vals + (long)B * M;
  // one query per warp: queries cost between one and several times the average, and a warp (or a block) that
  // takes several of them makes the last wave longer (8 per warp: 298 us instead of 232 us at 163 842 x 163 842)
  const dim3 grid((unsigned)((N + KNNT_WARPS - 1) / KNNT_WARPS), (unsigned)B);
  knn_tree_kernel<DT><<<grid, KNNT_WARPS * 32, 0, st>>>(query, M, N, k, L.nleaf, L.nnode, L.ngroup, keys,
                                                        qkeys, qvals, leaves, lbox, nbox, gbox, todo, listed, list,
                                                        budget, idx, dist), MC_COUNT(1);
  knn_thread_launch<DT>(ref, query, B, DT, M, N, k, idx, dist, st, todo);
  MC_CHECK_LAUNCH();
  return MC_OK;
}

// All pairs: up to how many queries a warp per query is the better choice.  It takes time for every pair, since each
// query loads the references again; a thread per query takes the same time for any number of queries that the chip
// holds.  Measured, in microseconds, warps / threads:
//   D = 3, 20 000 references:  16 000 queries 494 / 582, 30 000 896 / 669;  160 000: 12 000 2984 / 3167, 16 000 3753 / 3167
//   D = 4, 20 000 references:  20 000 queries 689 / 693;                    160 000:  8 000 2219 / 3312, 12 000 3374 / 3308
//   D = 8,  2 000 references:  20 000 queries 208 / 269, 30 000 312 / 269;  160 000: 12 000 9234 / 11280, 16 000 11659 / 11282
//   D = 16, 2 000 references:   8 000 queries 210 / 261, 12 000 320 / 263;  160 000:  2 000 5018 / 11420,  5 000 13843 / 11431
static long knn_few(int D, int M) {
  const double pair = D <= 4 ? 1.05e-3 + 0.15e-3 * D : D <= 8 ? 0.57e-3 * D : 0.95e-3 * D;  // ns
  const double threads = D <= 4 ? 150e3 + 20. * M : 130e3 + 70. * M;                        // ns
  return (long)(threads / (1.9 + pair * M));
}

// one thread per query; behind the search as many blocks as the chip holds, for the case of a warp per query
static int knn_blocks(int N, int threads, const KnnTodo& todo) {
  const int n = (N + threads - 1) / threads;
  return todo.crowded && n < 148 * 8 ? 148 * 8 : n;
}
template <int DT>
static void knn_thread_launch(const float* ref, const float* query, int B, int D, int M, int N, int k,
                              int64_t* idx, float* dist, cudaStream_t st, const KnnTodo& todo) {
  if (DT > 0 && k <= 16) {
    constexpr int DS = DT > 0 ? DT : 1;
    dim3 grid((unsigned)knn_blocks(N, KNN2_THREADS, todo), (unsigned)B);
    if (k <= 8) knn_small_d_kernel<DS, 8><<<grid, KNN2_THREADS, 0, st>>>(ref, query, M, N, k, idx, dist, todo), MC_COUNT(1);
    else if (k <= 12) knn_small_d_kernel<DS, 12><<<grid, KNN2_THREADS, 0, st>>>(ref, query, M, N, k, idx, dist, todo), MC_COUNT(1);
    else knn_small_d_kernel<DS, 16><<<grid, KNN2_THREADS, 0, st>>>(ref, query, M, N, k, idx, dist, todo), MC_COUNT(1);
    return;
  }
  dim3 grid((unsigned)knn_blocks(N, KNN_THREADS, todo), (unsigned)B);
  if (k <= 8) knn_kernel<DT, 8><<<grid, KNN_THREADS, 0, st>>>(ref, query, D, M, N, k, idx, dist, todo), MC_COUNT(1);
  else if (k <= 16) knn_kernel<DT, 16><<<grid, KNN_THREADS, 0, st>>>(ref, query, D, M, N, k, idx, dist, todo), MC_COUNT(1);
  else knn_kernel<DT, 32><<<grid, KNN_THREADS, 0, st>>>(ref, query, D, M, N, k, idx, dist, todo), MC_COUNT(1);
}

template <int DT>
static void knn_brute_launch(const float* ref, const float* query, int B, int D, int M, int N, int k,
                             int64_t* idx, float* dist, cudaStream_t st) {
  const long queries = (long)B * N;
  if (queries > knn_few(D, M)) {
    knn_thread_launch<DT>(ref, query, B, D, M, N, k, idx, dist, st, KnnTodo{});
    return;
  }
  const int wpq = knn_warps_per_query(queries, M, KNNW_MAX_WARPS);
  const int warps = wpq > KNNW_WARPS ? wpq : KNNW_WARPS, qpb = warps / wpq;
  knn_wide_kernel<DT><<<dim3((unsigned)((N + qpb - 1) / qpb), (unsigned)B), warps * 32, 0, st>>>(
      ref, query, D, M, N, k, idx, dist), MC_COUNT(1);
}

static int knn_check(const void* ref, const void* query, int B, int D, int M, int N, int k, const void* idx,
                     const void* dist) {
  if (!ref || !query || !idx || !dist) return MC_ERR_BAD_ARG;
  if (B <= 0 || D <= 0 || M <= 0 || N <= 0 || k <= 0) return MC_ERR_BAD_ARG;
  if (k > 32 || D > KNN_DMAX || B > 65535) return MC_ERR_TOO_LARGE;
  if (k > M) return MC_ERR_BAD_ARG;
  return MC_OK;
}

static bool knn_tree_shape(int B, int D, int M, int N) {
  return D <= KNNT_DMAX && B <= 128 && (long)B * ((long)M + N) < (1L << 30);
}

}  // namespace mc

using namespace mc;

extern "C" int mc_knn(const float* ref, const float* query, int32_t B, int32_t D, int32_t M,
                      int32_t N, int32_t k, int64_t* idx, float* dist, void* stream) {
  const int rc = knn_check(ref, query, B, D, M, N, k, idx, dist);
  if (rc) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  switch (D) {
    case 1: knn_brute_launch<1>(ref, query, B, D, M, N, k, idx, dist, st); break;
    case 2: knn_brute_launch<2>(ref, query, B, D, M, N, k, idx, dist, st); break;
    case 3: knn_brute_launch<3>(ref, query, B, D, M, N, k, idx, dist, st); break;
    case 4: knn_brute_launch<4>(ref, query, B, D, M, N, k, idx, dist, st); break;
    default: knn_brute_launch<0>(ref, query, B, D, M, N, k, idx, dist, st); break;
  }
  MC_CHECK_LAUNCH();
  return MC_OK;
}

// Sorting and building the leaves take about 60 us in a dozen launches, so the search pays from some number
// of pairs on (measured: 30 000 x 2 000 points 121 us against 133 us of all pairs, 10 000 x 3 000 109 us
// against 88 us, 163 842 x 163 842 0.31 ms against 7.65 ms).
constexpr double KNN_TREE_PAIRS = 5e7;

extern "C" size_t mc_knn_workspace_bytes(int32_t B, int32_t D, int32_t M, int32_t N, int32_t k) {
  if (B <= 0 || D <= 0 || M <= 0 || N <= 0 || k <= 0 || k > 32 || !knn_tree_shape(B, D, M, N)) return 0;
  if ((double)B * M * N < KNN_TREE_PAIRS || M < 32 * KNNT_LEAF) return 0;
  return knn_tree_layout(B, D, M, N, false).total;
}

extern "C" int mc_knn_ws(const float* ref, const float* query, int32_t B, int32_t D, int32_t M, int32_t N,
                         int32_t k, int64_t* idx, float* dist, void* ws, size_t ws_bytes, void* stream) {
  if (!ws) return mc_knn(ref, query, B, D, M, N, k, idx, dist, stream);
  const int rc = knn_check(ref, query, B, D, M, N, k, idx, dist);
  if (rc) return rc;
  if (!knn_tree_shape(B, D, M, N)) return MC_ERR_UNSUPPORTED;
  cudaStream_t st = (cudaStream_t)stream;
  switch (D) {
    case 1: return knn_tree_launch<1>(ref, query, B, M, N, k, idx, dist, ws, ws_bytes, st);
    case 2: return knn_tree_launch<2>(ref, query, B, M, N, k, idx, dist, ws, ws_bytes, st);
    default: return knn_tree_launch<3>(ref, query, B, M, N, k, idx, dist, ws, ws_bytes, st);
  }
}
