// ReduceSumOp / ReduceMaxOp for sm_100a.
//
// The tensor is viewed as A x B x C (row-major) and B is reduced, as the
// reference does (reduction/reduce_impl.h:28-59).  Both shapes of the problem
// are bound by HBM bandwidth, so every path is built around 128-bit coalesced
// streaming loads with several loads in flight per thread:
//
//   C == 1  ("rows"):    a group of 1..256 threads owns one row (or one segment
//                        of a long row); warp shuffles, then shared memory,
//                        combine the group.  Long rows with few rows in total are
//                        cut into segments: up to 8 segments are combined inside
//                        one thread-block cluster through distributed shared
//                        memory (single launch, no workspace); more segments go
//                        through f32 partials in the workspace and a second pass.
//   C  > 1  ("columns"): few rows, or columns enough for a thread each, are walked
//                        over by one thread per vector; otherwise threads sum
//                        super-rows (as many rows as make whole vectors) and B is
//                        split over enough blocks to fill 148 SMs.  Up to eight
//                        splits fold through distributed shared memory; more leave
//                        f32 partials, which a second pass folds in split order, so
//                        that the result does not depend on scheduling.  (Folding in
//                        the first launch - the last block of a slab to finish, found
//                        by a ticket, folds it - was measured slower: 14.4 against
//                        13.6 us on f16 [32768, 1024], because the fence, the ticket
//                        and the fold are one more latency chain after the last load,
//                        while the second pass is already resident and waiting.)
//
// Max semantics (reduction_helper.h:159-180 folded in ascending index order):
// NaN wins; otherwise the largest value; between +0 and -0, which compare equal,
// the one at the higher index.  The streaming pass uses the hardware max (which
// ranks -0 below +0); only a result that is exactly zero triggers a short
// backward scan for the last zero of the range to fix the sign.
#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace b200 {
namespace {

constexpr int kSum = B200_REDUCE_SUM;
constexpr int kMax = B200_REDUCE_MAX;
constexpr int kBlock = 256;
constexpr int kFinalizeBlock = 1024; // second pass: 32 outputs x 32 slices

__device__ __forceinline__ float max_nan_f32(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

template <int OP> __device__ __forceinline__ float op_init() {
  return OP == kSum ? 0.f : -INFINITY;
}
// order-insensitive combine of two partial results (zero signs fixed up later)
template <int OP> __device__ __forceinline__ float op_combine(float a, float b) {
  return OP == kSum ? a + b : max_nan_f32(a, b);
}
// the reference's apply(lhs, rhs) with lhs covering the lower indices
template <int OP> __device__ __forceinline__ float op_apply_ordered(float lhs, float rhs) {
  if (OP == kSum)
    return lhs + rhs;
  return (isnan(lhs) || lhs > rhs) ? lhs : rhs;
}

// ---- per-thread accumulators over 16-byte vectors --------------------------
template <typename T, int OP> struct Acc;

template <> struct Acc<float, kSum> {
  float a = 0.f, b = 0.f;
  __device__ __forceinline__ void vec(uint4 v) {
    a += __uint_as_float(v.x);
    b += __uint_as_float(v.y);
    a += __uint_as_float(v.z);
    b += __uint_as_float(v.w);
  }
  __device__ __forceinline__ void one(float v) { a += v; }
  __device__ __forceinline__ float get() const { return a + b; }
};
template <> struct Acc<float, kMax> {
  float m = -INFINITY;
  __device__ __forceinline__ void vec(uint4 v) {
    m = max_nan_f32(m, max_nan_f32(max_nan_f32(__uint_as_float(v.x), __uint_as_float(v.y)),
                                   max_nan_f32(__uint_as_float(v.z), __uint_as_float(v.w))));
  }
  __device__ __forceinline__ void one(float v) { m = max_nan_f32(m, v); }
  __device__ __forceinline__ float get() const { return m; }
};
template <> struct Acc<__half, kSum> {
  float a = 0.f, b = 0.f;
  __device__ __forceinline__ void word(uint32_t w) {
    float2 f = __half22float2(*reinterpret_cast<__half2 *>(&w));
    a += f.x;
    b += f.y;
  }
  __device__ __forceinline__ void vec(uint4 v) {
    word(v.x), word(v.y), word(v.z), word(v.w);
  }
  __device__ __forceinline__ void one(__half v) { a += __half2float(v); }
  __device__ __forceinline__ float get() const { return a + b; }
};
template <> struct Acc<__nv_bfloat16, kSum> {
  float a = 0.f, b = 0.f;
  __device__ __forceinline__ void word(uint32_t w) {
    a += __uint_as_float(w << 16);
    b += __uint_as_float(w & 0xffff0000u);
  }
  __device__ __forceinline__ void vec(uint4 v) {
    word(v.x), word(v.y), word(v.z), word(v.w);
  }
  __device__ __forceinline__ void one(__nv_bfloat16 v) { a += __bfloat162float(v); }
  __device__ __forceinline__ float get() const { return a + b; }
};
template <> struct Acc<__half, kMax> {
  __half2 m = __half2half2(__ushort_as_half((unsigned short)0xfc00)); // -inf
  __device__ __forceinline__ void word(uint32_t w) {
    m = __hmax2_nan(m, *reinterpret_cast<__half2 *>(&w));
  }
  __device__ __forceinline__ void vec(uint4 v) {
    word(v.x), word(v.y), word(v.z), word(v.w);
  }
  __device__ __forceinline__ void one(__half v) { m = __hmax2_nan(m, __half2half2(v)); }
  __device__ __forceinline__ float get() const {
    return max_nan_f32(__low2float(m), __high2float(m));
  }
};
template <> struct Acc<__nv_bfloat16, kMax> {
  __nv_bfloat162 m = __bfloat162bfloat162(__ushort_as_bfloat16((unsigned short)0xff80)); // -inf
  __device__ __forceinline__ void word(uint32_t w) {
    m = __hmax2_nan(m, *reinterpret_cast<__nv_bfloat162 *>(&w));
  }
  __device__ __forceinline__ void vec(uint4 v) {
    word(v.x), word(v.y), word(v.z), word(v.w);
  }
  __device__ __forceinline__ void one(__nv_bfloat16 v) {
    m = __hmax2_nan(m, __bfloat162bfloat162(v));
  }
  __device__ __forceinline__ float get() const {
    return max_nan_f32(__low2float(m), __high2float(m));
  }
};

template <typename OutT> __device__ __forceinline__ void store_out(OutT *p, float v) {
  *p = Elt<OutT>::from_f32(v);
}

// elements from p to the next 16-byte boundary
template <typename T> __device__ __forceinline__ int elements_to_boundary(const T *p) {
  return (int)((16 - (reinterpret_cast<uintptr_t>(p) & 15)) & 15) / (int)sizeof(T);
}

// =============================================================================
// rows: C == 1
// =============================================================================
// Grid: one group of `tpr` threads per (row, segment); kBlock / tpr groups per
// block.  kCluster: the `segs` blocks of a row form one cluster (tpr == kBlock).
// VEC: every row starts on a 16-byte boundary.  Otherwise each row has up to N - 1 elements in
// front of its first whole vector and as many behind its last; the group takes those one by one
// (tpr >= 2 N) and the rest in vectors.  (Element by element, f32 [4001, 4001] took 21.2 us.)
template <typename T, int OP, bool VEC, bool kCluster, typename OutT>
__global__ void __launch_bounds__(kBlock, 4)
    reduce_rows_kernel(const T *__restrict__ in, OutT *__restrict__ out,
                       float *__restrict__ partial, int64_t A, int64_t B, int tpr,
                       int segs, int64_t seg_len) {
  constexpr int N = 16 / sizeof(T);
  __shared__ float warp_part[kBlock / 32];
  __shared__ float cluster_part;
  pdl_launch_dependents();

  const int groups_per_block = kBlock / tpr;
  const int64_t g = (int64_t)blockIdx.x * groups_per_block + threadIdx.x / tpr;
  const int t = threadIdx.x % tpr;
  const int64_t a = g / segs;
  const int s = (int)(g % segs);
  const bool active = a < A;
  const int64_t e0 = (int64_t)s * seg_len;
  const int64_t e1 = active ? min(B, e0 + seg_len) : e0;
  const T *row = in + (active ? a : 0) * B;

  // elements in front of the first 16-byte boundary (rows whose length is no multiple of 16 bytes start anywhere)
  const int head = (int)min(e1 - e0, (int64_t)(VEC ? 0 : elements_to_boundary(row + e0)));
  const uint4 *vp = reinterpret_cast<const uint4 *>(row + e0 + head);
  const int64_t nvec = (e1 - e0 - head) / N;
  { // the first loads, on their way into L2 while the kernel in front of this one ends
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (t + (int64_t)k * tpr < nvec)
        prefetch_l2(vp + t + (int64_t)k * tpr);
  }
  pdl_wait();
  Acc<T, OP> acc;
  if (!VEC) { // the edges, fewer than 2 N <= tpr elements, requested in front of the vectors
    const int edges = head + (int)(e1 - e0 - head - nvec * N);
    if (t < edges)
      acc.one(row[e0 + (t < head ? (int64_t)t : nvec * N + t)]);
  }
  // eight loads in flight per thread, the last batch predicated: one memory latency per batch
  for (int64_t v = t; v < nvec; v += 8 * (int64_t)tpr) {
    uint4 x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (v + u * (int64_t)tpr < nvec)
        x[u] = ld_nc_v4(vp + v + u * (int64_t)tpr);
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (v + u * (int64_t)tpr < nvec)
        acc.vec(x[u]);
  }
  if (VEC)
    for (int64_t e = e0 + nvec * N + t; e < e1; e += tpr)
      acc.one(row[e]);
  float r = acc.get();

  // combine the group; every thread of the group ends up with the result
  const int width = tpr < 32 ? tpr : 32;
  for (int off = width >> 1; off > 0; off >>= 1)
    r = op_combine<OP>(r, __shfl_xor_sync(0xffffffffu, r, off));
  if (tpr > 32) {
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0)
      warp_part[warp] = r;
    __syncthreads();
    const int w0 = (threadIdx.x / tpr) * (tpr >> 5);
    r = warp_part[w0];
    for (int w = 1; w < (tpr >> 5); ++w)
      r = op_combine<OP>(r, warp_part[w0 + w]);
  }

  // max == 0: the sign is that of the last zero of the range
  if (OP == kMax && active && r == 0.f) {
    const int lanes = width; // the first `width` threads of the group scan backwards
    const unsigned gmask =
        tpr >= 32 ? 0xffffffffu : (((1u << tpr) - 1u) << ((threadIdx.x & 31) / tpr * tpr));
    if (t < lanes) {
      float found = 0.f;
      for (int64_t hi = e1; hi > e0; hi -= lanes) {
        const int64_t e = hi - 1 - t;
        const float v = e >= e0 ? Elt<T>::to_f32(row[e]) : 1.f;
        const unsigned hit = __ballot_sync(gmask, v == 0.f);
        if (hit) {
          // lowest t = highest index
          const int src = __ffs(hit) - 1;
          found = __shfl_sync(gmask, v, src);
          break;
        }
      }
      r = found; // thread t == 0, which writes the result, is one of the scanners
    }
  }

  if (kCluster) {
    cg::cluster_group cluster = cg::this_cluster();
    if (threadIdx.x == 0)
      cluster_part = r;
    cluster.sync();
    if (cluster.block_rank() == 0 && threadIdx.x == 0) {
      float total = r;
      for (int k = 1; k < segs; ++k)
        total = op_apply_ordered<OP>(total, *cluster.map_shared_rank(&cluster_part, k));
      store_out(out + a, total);
    }
    cluster.sync(); // keep every block's shared memory alive until rank 0 has read it
    return;
  }
  if (active && t == 0) {
    if (segs == 1)
      store_out(out + a, r);
    else
      partial[a * segs + s] = r;
  }
}

// Short rows (a row is at most VPT 16-byte vectors per thread of its group):
// persistent blocks walk over the rows, and the loads of the next row are issued
// before the current one is reduced, so that every thread keeps VPT..2*VPT loads
// in flight across row boundaries.  VEC as above.
template <typename T, int OP, int VPT, bool VEC, typename OutT>
__global__ void __launch_bounds__(kBlock)
    reduce_short_rows_kernel(const T *__restrict__ in, OutT *__restrict__ out, int64_t A, int64_t B,
                             int tpr, int prefetch) {
  constexpr int N = 16 / sizeof(T);
  __shared__ float warp_part[2][kBlock / 32];
  pdl_launch_dependents();
  const int groups_per_block = kBlock / tpr;
  const int t = threadIdx.x % tpr;
  const int gib = threadIdx.x / tpr;
  const int64_t block_rows = groups_per_block;
  const int64_t iters = ceil_div<int64_t>(ceil_div<int64_t>(A, block_rows) - blockIdx.x, (int64_t)gridDim.x);
  const int width = tpr < 32 ? tpr : 32;

  struct Row {
    uint4 v[VPT];
    T edge;       // one of the elements in front of the first or behind the last vector
    int nvec, edges;
  };
  Row cur, nxt;
  auto load_row = [&](int64_t a, Row &r) {
    const T *p = in + a * B;
    const int head = VEC ? 0 : min((int)B, elements_to_boundary(p));
    r.nvec = a < A ? (int)(B - head) / N : 0;
    const uint4 *vp = reinterpret_cast<const uint4 *>(p + head);
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int idx = t + k * tpr;
      if (idx < r.nvec)
        r.v[k] = ld_nc_v4(vp + idx);
    }
    if (!VEC) {
      r.edges = a < A ? (int)B - r.nvec * N : 0;
      if (t < r.edges)
        r.edge = p[t < head ? t : r.nvec * N + t];
    }
  };
  int64_t a = (int64_t)blockIdx.x * block_rows + gib;
  // the loads of the first `prefetch` rows of this group, on their way into L2 during the wait
  for (int64_t ap = a, k = 0; k < prefetch && ap < A; ++k, ap += (int64_t)gridDim.x * block_rows) {
    const T *p = in + ap * B;
#pragma unroll
    for (int k2 = 0; k2 < VPT; ++k2)
      if (t + k2 * tpr < (int)(B / N))
        prefetch_l2(p + (t + k2 * tpr) * N);
  }
  pdl_wait();
  load_row(a, cur);
  for (int64_t it = 0; it < iters; ++it) {
    const int64_t a_next = a + (int64_t)gridDim.x * block_rows;
    if (it + 1 < iters)
      load_row(a_next, nxt);
    const bool active = a < A;
    Acc<T, OP> acc;
#pragma unroll
    for (int k = 0; k < VPT; ++k)
      if (t + k * tpr < cur.nvec)
        acc.vec(cur.v[k]);
    if (!VEC && t < cur.edges)
      acc.one(cur.edge);
    float r = acc.get();
    for (int off = width >> 1; off > 0; off >>= 1)
      r = op_combine<OP>(r, __shfl_xor_sync(0xffffffffu, r, off));
    if (tpr > 32) {
      float *wp = warp_part[it & 1];
      if ((threadIdx.x & 31) == 0)
        wp[threadIdx.x >> 5] = r;
      __syncthreads();
      const int w0 = gib * (tpr >> 5);
      r = wp[w0];
      for (int w = 1; w < (tpr >> 5); ++w)
        r = op_combine<OP>(r, wp[w0 + w]);
    }
    if (OP == kMax && active && r == 0.f) { // sign of the last zero of the row
      const unsigned gmask =
          tpr >= 32 ? 0xffffffffu : (((1u << tpr) - 1u) << ((threadIdx.x & 31) / tpr * tpr));
      if (t < width) {
        const T *row = in + a * B;
        float found = 0.f;
        for (int64_t hi = B; hi > 0; hi -= width) {
          const int64_t e = hi - 1 - t;
          const float v = e >= 0 ? Elt<T>::to_f32(row[e]) : 1.f;
          const unsigned hit = __ballot_sync(gmask, v == 0.f);
          if (hit) {
            found = __shfl_sync(gmask, v, __ffs(hit) - 1);
            break;
          }
        }
        r = found;
      }
    }
    if (active && t == 0)
      store_out(out + a, r);
    cur = nxt;
    a = a_next;
  }
}

// Short rows that start off the 16-byte boundary: `rows` neighbouring rows are one contiguous piece of memory, which
// the block brings into shared memory in 16-byte vectors (its own first and last elements one by one); then `tpr`
// threads sum each row from there.  Groups that read such rows from global memory have a handful of loads in flight
// per warp and most lanes idle: f16 [1000000, 33] took 28 us element by element and 137 us in vectors per row.
constexpr int kChunkBytes = 16384;
constexpr int kChunkRow = 256; // longest row; above, a group of lanes per row is faster (f16 [100000, 255]: 13 against 20 us)
template <typename T, int OP, typename OutT>
__global__ void __launch_bounds__(kBlock)
    reduce_chunk_rows_kernel(const T *__restrict__ in, OutT *__restrict__ out, int64_t A, int B, int tpr, int rows) {
  constexpr int N = 16 / sizeof(T);
  __shared__ __align__(16) T sm[kChunkBytes / sizeof(T) + N];
  pdl_launch_dependents();
  const int64_t a0 = (int64_t)blockIdx.x * rows;
  const int here = (int)min((int64_t)rows, A - a0), count = here * B;
  const T *p = in + a0 * B;
  const int head = min(count, elements_to_boundary(p)), nvec = (count - head) / N;
  T *dst = sm + (N - head) % N; // the first whole vector lands on a 16-byte boundary
  const uint4 *vp = reinterpret_cast<const uint4 *>(p + head);
  for (int v = threadIdx.x; v < nvec; v += kBlock)
    prefetch_l2(vp + v);
  pdl_wait();
  const int edges = count - nvec * N;
  if (threadIdx.x < edges) {
    const int e = threadIdx.x < head ? threadIdx.x : nvec * N + threadIdx.x;
    dst[e] = p[e];
  }
#pragma unroll 4
  for (int v = threadIdx.x; v < nvec; v += kBlock)
    *reinterpret_cast<uint4 *>(dst + head + v * N) = ld_nc_v4(vp + v);
  __syncthreads();
  const int t = threadIdx.x % tpr, groups = kBlock / tpr;
  for (int r = threadIdx.x / tpr; r - (int)(threadIdx.x / tpr) < here; r += groups) { // every thread runs every turn: shuffles
    const T *row = dst + min(r, here - 1) * B;
    float x = op_init<OP>(), y = op_init<OP>();
    int e = t;
    for (; e + tpr < B; e += 2 * tpr) {
      x = op_combine<OP>(x, Elt<T>::to_f32(row[e]));
      y = op_combine<OP>(y, Elt<T>::to_f32(row[e + tpr]));
    }
    if (e < B)
      x = op_combine<OP>(x, Elt<T>::to_f32(row[e]));
    x = op_combine<OP>(x, y);
    for (int off = tpr >> 1; off > 0; off >>= 1)
      x = op_combine<OP>(x, __shfl_xor_sync(0xffffffffu, x, off));
    if (t == 0 && r < here) {
      if (OP == kMax && x == 0.f) { // the sign of the last zero of the row
        for (int k = B - 1; k >= 0; --k) {
          const float v = Elt<T>::to_f32(row[k]);
          if (v == 0.f) {
            x = v;
            break;
          }
        }
      }
      store_out(out + a0 + r, x);
    }
  }
}

// =============================================================================
// columns: C > 1
// =============================================================================
// One matrix (one a) is a run of B * C elements, and what a 16-byte vector of it holds repeats
// every P rows, where P * C elements are a multiple of 16 bytes: a "super-row" of P rows.  The
// kernel sums super-rows, so every load is a whole vector whatever C is (element by element, f16
// [32768, 1023] took 32 us and [64, 50000, 3] 15 us).  Up to N - 1 elements in front of the first
// 16-byte boundary and the part of a super-row at the end are taken one by one; the first super-row
// starts at the boundary, `head` elements into the run, so position i of a super-row belongs to
// column (head + i) mod C.
//
// A block covers `lpr` threads x VPT vectors of the super-row (a slab) and `row_lanes` super-rows at
// a time.  Where the slab is the whole super-row the block also folds its P rows; otherwise (C of
// more than 1024 vectors per P rows) the P rows of a column lie in different slabs and the second
// pass folds them.  The B rows are split over blocks, either the blocks of a cluster (CLUSTER),
// which fold through distributed shared memory, or blocks whose partial sums a second pass folds.
// Bound by memory from ~64 MB on, by the latency of one or two launches below.  Before / now, us: bf16 max
// [64, 1000, 129] 12.7 / 7.3, f16 [32768, 1023] 32 / 20, bf16 [2, 100000, 300] 54 / 23 (5.2 TB/s), f32 [1000, 16384]
// 15.7 / 11.6 (5.7 TB/s).
struct ColsPlan {
  int64_t P;             // rows of a super-row
  int64_t nvec;          // its vectors
  int vpt, lpr, row_lanes, threads;
  int slabs, splits;
  int64_t supers_per_split;
  bool cluster;
  bool fold_rows;        // slabs == 1: the block folds the P rows
};

template <typename T, int OP> struct Vec16 {
  static constexpr int N = 16 / sizeof(T);
  static __device__ __forceinline__ void add(float (&acc)[N], const uint4 &v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if constexpr (sizeof(T) == 4) {
        acc[k] = op_combine<OP>(acc[k], __uint_as_float(w[k]));
      } else {
        float lo, hi;
        if constexpr (std::is_same<T, __half>::value) {
          float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&w[k]));
          lo = f.x, hi = f.y;
        } else {
          lo = __uint_as_float(w[k] << 16);
          hi = __uint_as_float(w[k] & 0xffff0000u);
        }
        acc[2 * k] = op_combine<OP>(acc[2 * k], lo);
        acc[2 * k + 1] = op_combine<OP>(acc[2 * k + 1], hi);
      }
    }
  }
};

// A maximum that is exactly zero takes the sign of the last zero of its column (the hardware max
// ranks -0 below +0): a backward scan of rows [lo, hi) that ends at that zero, LOADS of them in flight.
template <int LOADS, typename T> __device__ __forceinline__ float scan_for_zero(const T *col, int64_t lo, int64_t hi, int64_t C) {
#pragma unroll 1
  for (int64_t r = hi - 1; r >= lo; r -= LOADS) {
    float v[LOADS];
#pragma unroll
    for (int u = 0; u < LOADS; ++u)
      v[u] = r - u >= lo ? Elt<T>::to_f32(col[(r - u) * C]) : 1.f;
#pragma unroll
    for (int u = 0; u < LOADS; ++u)
      if (v[u] == 0.f)
        return v[u];
  }
  return 0.f;
}
// Out of line: it is rare, and its registers cost the two kernels that use it blocks per SM.  (The kernels of super-rows, at
// their limit of 64 registers, are 10 % slower with a call in them.)
template <typename T> __device__ __noinline__ float last_zero(const T *col, int64_t hi, int64_t C) {
  return scan_for_zero<16>(col, 0, hi, C);
}
// The same where the rows are split over blocks: the last zero lies in the rows of the last split whose maximum is zero, and
// only those are scanned (all rows, one by one, of f16 [32768, 1024] with one zero in front took 7.1 ms a call, now 52 us).  `run`: the
// matrix, `split`: that split, `split_elems`: the elements of one, the last one's end `super` or fewer behind it.
template <typename T>
__device__ __forceinline__ float last_zero_of_split(const T *run, int64_t c, int split, int splits, int64_t split_elems, int64_t super, int64_t B,
                                    int64_t C) {
  const int64_t total = B * C, head = min(total, (int64_t)elements_to_boundary(run));
  const int64_t begin = split == 0 ? 0 : max((int64_t)0, min(head + split * split_elems, total - super));
  const int64_t end = split == splits - 1 ? total : min(total, head + (split + 1) * split_elems);
  return scan_for_zero<8>(run + c, begin / C, min(B, (end + C - 1) / C), C); // a row too many on either side changes nothing
}

template <typename T, int OP, int VPT, bool CLUSTER, typename OutT>
__global__ void __launch_bounds__(512, 2)
    reduce_cols_kernel(const T *__restrict__ in, OutT *__restrict__ out, float *__restrict__ partial, int64_t A, int64_t B,
                       int64_t C, const __grid_constant__ ColsPlan p, int prefetch) {
  constexpr int N = 16 / sizeof(T);
  constexpr int U = 8 / VPT; // super-rows per batch: eight loads in flight per thread
  extern __shared__ float sums[]; // [row lane][position of the slab], then folded
  pdl_launch_dependents(); // lets the next kernel (the second pass) be scheduled while this one runs

  const int64_t bid = blockIdx.x;
  int slab, split;
  int64_t a;
  if (CLUSTER) { // the splits of one (a, slab) are neighbours
    split = (int)(bid % p.splits);
    slab = (int)(bid / p.splits % p.slabs);
    a = bid / p.splits / p.slabs;
  } else {
    slab = (int)(bid % p.slabs);
    split = (int)(bid / p.slabs % p.splits);
    a = bid / p.slabs / p.splits;
  }
  const T *run = in + a * B * C;
  const int64_t super = p.P * C, total = B * C;
  const int head = (int)min(total, (int64_t)elements_to_boundary(run));
  const int64_t supers = (total - head) / super;
  const int64_t s0 = (int64_t)split * p.supers_per_split;
  const int64_t s1 = split == p.splits - 1 ? supers : min(supers, s0 + p.supers_per_split);
  const int lane_row = threadIdx.x / p.lpr, lane_col = threadIdx.x - lane_row * p.lpr;
  const int64_t first_vec = (int64_t)slab * p.lpr * VPT; // of the slab
  const T *base = run + head + (first_vec + lane_col) * N;
  bool ok[VPT];
#pragma unroll
  for (int k = 0; k < VPT; ++k)
    ok[k] = lane_row < p.row_lanes && first_vec + lane_col + (int64_t)k * p.lpr < p.nvec;
  const int64_t step = (int64_t)p.row_lanes * super; // elements between the super-rows of a thread
  const int kstep = p.lpr * N;
  const int mine = (int)((s1 - s0 - lane_row + p.row_lanes - 1) / p.row_lanes); // super-rows of this thread (or <= 0)
  const T *q = base + (s0 + lane_row) * super;
  {
    // the first batches of this thread's loads, on their way into L2 during the wait
    const T *f = q;
    for (int i = 0; i < prefetch * U && i < mine; ++i, f += step)
#pragma unroll
      for (int k = 0; k < VPT; ++k)
        if (ok[k])
          prefetch_l2(f + k * kstep);
  }
  pdl_wait(); // inputs may come from the kernel launched just before this one

  float acc[VPT][N];
#pragma unroll
  for (int k = 0; k < VPT; ++k)
#pragma unroll
    for (int j = 0; j < N; ++j)
      acc[k][j] = op_init<OP>();
  // the last, partial batch is predicated rather than handled load by load, so the tail does not pay
  // one memory latency per row
  for (int i = 0; i < mine; i += U) {
    uint4 x[U][VPT];
#pragma unroll
    for (int u = 0; u < U; ++u, q += step)
#pragma unroll
      for (int k = 0; k < VPT; ++k)
        if (ok[k] && i + u < mine)
          x[u][k] = ld_nc_v4(q + k * kstep);
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int k = 0; k < VPT; ++k)
        if (ok[k] && i + u < mine)
          Vec16<T, OP>::add(acc[k], x[u][k]);
  }
  if (lane_row == 0) {
    // what is left at the end goes to the last split, the elements in front of the boundary to the
    // first (they are the last `head` positions of the super-row in front)
    const int64_t rest = split == p.splits - 1 ? total - head - supers * super : 0;
    const int64_t front = split == 0 ? super - head : super;
    const T *end = run + head + supers * super;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int64_t i0 = (first_vec + lane_col + (int64_t)k * p.lpr) * N;
      if (ok[k] && i0 + N <= rest)
        Vec16<T, OP>::add(acc[k], ld_nc_v4(end + i0));
      if (ok[k] && ((i0 < rest && i0 + N > rest) || i0 + N > front))
#pragma unroll
        for (int j = 0; j < N; ++j) {
          if (i0 + N > rest && i0 + j < rest)
            acc[k][j] = op_combine<OP>(acc[k][j], Elt<T>::to_f32(end[i0 + j]));
          if (i0 + j >= front)
            acc[k][j] = op_combine<OP>(acc[k][j], Elt<T>::to_f32(run[i0 + j - front]));
        }
    }
  }
  // rows of `width` sums, folded in halves down to one row: positions that are C apart where the slab
  // is the whole super-row, the row lanes otherwise
  const int slab_width = p.fold_rows ? (int)super : p.lpr * VPT * N;
#pragma unroll
  for (int k = 0; k < VPT; ++k)
    if (ok[k]) {
      float *dst = sums + lane_row * slab_width + (lane_col + k * p.lpr) * N;
#pragma unroll
      for (int j = 0; j < N; ++j)
        dst[j] = acc[k][j];
    }
  __syncthreads();
  const int width = p.fold_rows ? (int)C : slab_width;
  int height = p.fold_rows ? p.row_lanes * (int)p.P : p.row_lanes;
  while (height > 1) {
    const int half = (height + 1) / 2, n = (height - half) * width;
    for (int i = threadIdx.x; i < n; i += blockDim.x)
      sums[i] = op_combine<OP>(sums[i], sums[i + half * width]);
    height = half;
    __syncthreads();
  }
  // position -> column
  const int64_t limit = p.fold_rows ? C : min((int64_t)slab_width, super - first_vec * N);
  auto column = [&](int i) {
    const int64_t c = (head + first_vec * N + i) % C;
    return c;
  };
  auto finish = [&](int i, float r, int last_with_zero) {
    const int64_t c = column(i);
    if (OP == kMax && r == 0.f)
      r = last_zero_of_split(run, c, last_with_zero, p.splits, p.supers_per_split * super, super, B, C);
    store_out(out + a * C + c, r);
  };
  if (CLUSTER) {
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    const int rank = (int)cluster.block_rank();
    for (int i = rank * (int)blockDim.x + threadIdx.x; i < limit; i += p.splits * (int)blockDim.x) {
      float v[8], r;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (k < p.splits)
          v[k] = *cluster.map_shared_rank(sums + i, k);
      r = v[0];
#pragma unroll
      for (int k = 1; k < 8; ++k)
        if (k < p.splits)
          r = op_combine<OP>(r, v[k]);
      int zero = 0;
      if (OP == kMax)
#pragma unroll
        for (int k = 1; k < 8; ++k)
          if (k < p.splits && v[k] == 0.f)
            zero = k;
      finish(i, r, zero);
    }
    cluster.sync(); // keep every block's shared memory alive until all have read it
    return;
  }
  for (int i = threadIdx.x; i < limit; i += blockDim.x) {
    if (p.splits == 1 && (p.fold_rows || p.P == 1))
      finish(i, sums[i], 0);
    else if (p.fold_rows)
      partial[((int64_t)split * A + a) * C + column(i)] = sums[i];
    else
      partial[((int64_t)split * A + a) * super + first_vec * N + i] = sums[i];
  }
}

// One thread per 16-byte vector of the output's columns (VEC), or per column, for all B rows: no fold, no barrier, eight
// loads in flight.  For few rows, and for so many columns that the threads fill the chip (see cols_plan).  The eight rows of a
// batch are folded in pairs, so that a sum's chain has B / 8 additions, as many as where eight warps share the rows.
template <typename T, int OP, bool VEC, typename OutT>
__global__ void __launch_bounds__(kBlock)
    reduce_cols_direct_kernel(const T *__restrict__ in, OutT *__restrict__ out, int64_t units, int64_t B, int64_t C, int64_t per_row,
                              FastDiv by_row) {
  constexpr int N = VEC ? 16 / sizeof(T) : 1;
  pdl_launch_dependents();
  const int64_t i = (int64_t)blockIdx.x * kBlock + threadIdx.x;
  const bool ok = i < units;
  const int64_t a = units < (1LL << 31) ? (int64_t)by_row.quot((uint32_t)i) : i / per_row;
  const T *p = in + (ok ? a * B * C + (i - a * per_row) * N : 0);
  if (ok)
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (u < B)
        prefetch_l2(p + u * C);
  pdl_wait();
  if (!ok)
    return;
  float acc[N];
#pragma unroll
  for (int j = 0; j < N; ++j)
    acc[j] = op_init<OP>();
  auto value = [](const auto &v, int j) -> float { // element j of a loaded unit
    if constexpr (!VEC) {
      return Elt<T>::to_f32(v);
    } else {
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
      if constexpr (sizeof(T) == 4)
        return __uint_as_float(w[j]);
      else if constexpr (std::is_same<T, __half>::value)
        return __half2float(__ushort_as_half((unsigned short)(w[j >> 1] >> (j & 1) * 16)));
      else
        return __uint_as_float(j & 1 ? w[j >> 1] & 0xffff0000u : w[j >> 1] << 16);
    }
  };
  for (int64_t r = 0; r < B; r += 8, p += 8 * C) {
    typename std::conditional<VEC, uint4, T>::type x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      if (r + u < B) {
        if constexpr (VEC)
          x[u] = ld_nc_v4(p + u * C);
        else
          x[u] = p[u * C];
      }
#pragma unroll
    for (int j = 0; j < N; ++j) {
      float s[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        s[u] = r + u < B ? value(x[u], j) : op_init<OP>();
#pragma unroll
      for (int half = 4; half > 0; half /= 2)
#pragma unroll
        for (int u = 0; u < half; ++u)
          s[u] = op_combine<OP>(s[u], s[u + half]);
      acc[j] = op_combine<OP>(acc[j], s[0]);
    }
  }
  if (OP == kMax)
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (acc[j] == 0.f)
        acc[j] = last_zero(in + a * B * C + (i - a * per_row) * N + j, B, C);
  OutT *o = out + i * N;
  if constexpr (VEC) {
    __align__(16) OutT v[N];
#pragma unroll
    for (int j = 0; j < N; ++j)
      v[j] = Elt<OutT>::from_f32(acc[j]);
#pragma unroll
    for (int k = 0; k < (int)(N * sizeof(OutT) / 16); ++k)
      reinterpret_cast<uint4 *>(o)[k] = reinterpret_cast<const uint4 *>(v)[k];
  } else {
    store_out(o, acc[0]);
  }
}

// Eight warps share the rows, element by element, four columns and four rows in flight per thread: where super-rows do not
// pay and there are too few columns for a thread each (see cols_plan).
constexpr int kScalarCols = 4;
template <typename T, int OP, typename OutT>
__global__ void __launch_bounds__(kBlock)
    reduce_cols_scalar_kernel(const T *__restrict__ in, OutT *__restrict__ out, int64_t A, int64_t B, int64_t C, int slabs) {
  __shared__ float sums[8][32 * kScalarCols];
  const int slab = blockIdx.x % slabs, lane = threadIdx.x & 31, row = threadIdx.x >> 5;
  const int64_t a = blockIdx.x / slabs, c0 = (int64_t)slab * (32 * kScalarCols);
  const T *run = in + a * B * C;
  pdl_launch_dependents();
  pdl_wait();
  float acc[kScalarCols];
#pragma unroll
  for (int k = 0; k < kScalarCols; ++k)
    acc[k] = op_init<OP>();
  for (int64_t r = row; r < B; r += 32) {
    T x[4][kScalarCols];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int k = 0; k < kScalarCols; ++k)
        if (r + 8 * u < B && c0 + lane + 32 * k < C)
          x[u][k] = run[(r + 8 * u) * C + c0 + lane + 32 * k];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int k = 0; k < kScalarCols; ++k)
        if (r + 8 * u < B && c0 + lane + 32 * k < C)
          acc[k] = op_combine<OP>(acc[k], Elt<T>::to_f32(x[u][k]));
  }
#pragma unroll
  for (int k = 0; k < kScalarCols; ++k)
    sums[row][lane + 32 * k] = acc[k];
  __syncthreads();
  const int i = threadIdx.x;
  if (i < 32 * kScalarCols && c0 + i < C) {
    float r = sums[0][i];
#pragma unroll
    for (int w = 1; w < 8; ++w)
      r = op_combine<OP>(r, sums[w][i]);
    if (OP == kMax && r == 0.f)
      r = last_zero(run + c0 + i, B, C);
    store_out(out + a * C + c0 + i, r);
  }
}

// second pass of the columns: folds the splits (and, where the slabs did not, the P rows of a super-row).
// 32 outputs per block; 32 warps each fold a slice of the partial sums with 8 loads in flight, then warp 0
// folds the slices in order.
template <typename T, int OP, typename OutT>
__global__ void __launch_bounds__(kFinalizeBlock)
    reduce_cols_fold_kernel(const float *__restrict__ partial, const T *__restrict__ in, OutT *__restrict__ out, int64_t A,
                            int64_t B, int64_t C, int P, int splits, bool rotated, int64_t split_elems, int64_t super_elems) {
  __shared__ float sm[kFinalizeBlock / 32][32];
  __shared__ int zeros[OP == kMax ? kFinalizeBlock / 32 : 1][32]; // the last partial result of a slice that is zero
  constexpr int kSlices = kFinalizeBlock / 32;
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int64_t n = A * C, i = (int64_t)blockIdx.x * 32 + lane;
  const int64_t a = i / C, c = i - a * C, super = P * C;
  const T *run = in + a * B * C;
  int64_t at = c; // position of the column in the super-row
  if (rotated) { // the partial sums lie in the order of the super-row, which starts at the 16-byte boundary
    at -= elements_to_boundary(run) % C;
    at += at < 0 ? C : 0;
  }
  const float *p = partial + a * super + at;
  const int64_t split_stride = A * super;
  const int count = splits * P, per = (count + kSlices - 1) / kSlices;
  const int s0 = slice * per, s1 = min(count, s0 + per);
  pdl_wait(); // the partials come from the kernel launched just before this one
  pdl_launch_dependents();
  float r = op_init<OP>();
  int zero = -1;
  if (i < n)
    for (int s = s0; s < s1; s += 8) { // one memory latency per batch, the last one predicated
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (s + u < s1) {
          const int split = P == 1 ? s + u : (s + u) / P, row = P == 1 ? 0 : s + u - split * P;
          v[u] = p[split * split_stride + row * C];
        }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (s + u < s1) {
          r = op_combine<OP>(r, v[u]);
          if (OP == kMax && v[u] == 0.f)
            zero = s + u;
        }
    }
  sm[slice][lane] = r;
  if (OP == kMax)
    zeros[slice][lane] = zero;
  __syncthreads();
  if (slice == 0 && i < n) {
    r = sm[0][lane];
    for (int w = 1; w < kSlices && w * per < count; ++w)
      r = op_combine<OP>(r, sm[w][lane]);
    if (OP == kMax && r == 0.f) {
      for (int w = 1; w < kSlices && w * per < count; ++w)
        zero = max(zero, zeros[w][lane]);
      r = last_zero_of_split(run, c, zero / P, splits, split_elems, super_elems, B, C);
    }
    store_out(out + i, r);
  }
}

// second pass: out[i] = fold over s of partial[i * stride_i + s * stride_s].
// 32 outputs per block; 32 warps each fold a contiguous slice of the `count`
// partials with 8 loads in flight, then warp 0 folds the slice results in order.
// (The second pass is a latency chain, not a bandwidth problem: with 8 warps and 4
// loads in flight it took a third as long as the first pass over 64 MB.)
template <int OP, typename OutT>
__global__ void __launch_bounds__(kFinalizeBlock)
    reduce_finalize_kernel(const float *__restrict__ partial, OutT *__restrict__ out,
                           int64_t n, int count, int64_t stride_i, int64_t stride_s) {
  __shared__ float sm[kFinalizeBlock / 32][32];
  pdl_wait(); // the partials come from the kernel launched just before this one
  pdl_launch_dependents();
  constexpr int kSlices = kFinalizeBlock / 32;
  const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * 32 + lane;
  const int per = (count + kSlices - 1) / kSlices;
  const int s0 = slice * per, s1 = min(count, s0 + per);
  float r = 0.f;
  if (i < n && s0 < s1) {
    const float *p = partial + i * stride_i;
    r = p[s0 * stride_s];
    // batches of eight loads in flight, the last one predicated: one memory latency per batch
    for (int s = s0 + 1; s < s1; s += 8) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (s + u < s1)
          v[u] = p[(s + u) * stride_s];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (s + u < s1)
          r = op_apply_ordered<OP>(r, v[u]);
    }
  }
  sm[slice][lane] = r;
  __syncthreads();
  if (slice == 0 && i < n) {
    r = sm[0][lane];
    for (int w = 1; w < kSlices && w * per < count; ++w)
      r = op_apply_ordered<OP>(r, sm[w][lane]);
    store_out(out + i, r);
  }
}

template <typename OutT>
__global__ void __launch_bounds__(kBlock)
    cast_from_f32_kernel(const float *__restrict__ in, OutT *__restrict__ out, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * kBlock + threadIdx.x;
  if (i < n)
    out[i] = Elt<OutT>::from_f32(in[i]);
}

// plan constants of the column path (threads that cover one row of a slab; blocks per SM aimed at)
constexpr int kColsThreadsPerRow = 32;
// Measurement override of the column plan (b200_reduce_cols_plan_override): threads per slab
// row (0 = the rule above).
int g_cols_lpr_override = 0;
// How many batches of eight loads (column kernel) and rows (short-row kernel) a thread hints into L2
// before it waits for the kernel in front of it, and how many blocks per SM the two kernels aim at
// (both use 64 registers per thread, so four blocks of 256 threads fill an SM: more would be a
// second wave).  Measured on f16 [64, 512, 1024] (us per op, graph replay): column sum 13.6 with one
// batch hinted, 14.1 with two, 15.3 with four, 14.4 with none; row max 12.5 with nothing hinted,
// 10.5 with one row, 10.2 with four; two or three column blocks per SM 16.4 / 15.5 against 13.6.
// b200_reduce_tune changes them for such measurements.
int g_prefetch_cols = 1;
int g_prefetch_rows = 4;
int g_cols_blocks_per_sm = 4;
int g_rows_blocks_per_sm = 4;
// Block slots of a one-wave grid that are left free (b200_reduce_reserve_blocks).  The column and the
// short-row kernels fill every SM exactly (4 blocks of 256 threads x 64 registers), so a small kernel
// that runs beside them, like the exchange of a sharded sum, would push blocks into a second wave.
int g_reserved_blocks = 0;

// ---- launch plan: a pure function of the shape -----------------------------
enum ColsPath { kSuper, kScalar, kDirect };
struct Plan {
  bool rows;
  // rows
  int tpr, segs;
  int64_t seg_len;
  bool cluster;
  // columns
  ColsPath path;
  ColsPlan cols;
  size_t ws_bytes;      // what the launch uses
  size_t declared_bytes; // what b200_reduce_workspace_bytes says
};

// The split of the B rows over blocks aims at one wave (four blocks of 256 threads per SM, 64 registers per thread)
// with at least four super-rows per thread.
void split_cols(ColsPlan &p, int64_t A, int64_t B) {
  const int64_t supers = std::max<int64_t>(1, B / p.P), blocks = A * p.slabs;
  const int64_t per_sm = std::max(1, g_cols_blocks_per_sm * kBlock / p.threads);
  const int64_t wave = std::max<int64_t>(1, per_sm * kNumSMs - g_reserved_blocks);
  // not more blocks than the wave holds, unless that leaves much of it empty
  int64_t splits = std::max<int64_t>(1, g_reserved_blocks > 0 || wave / blocks >= 3 ? wave / blocks : ceil_div<int64_t>(wave, blocks));
  splits = std::min<int64_t>(splits, std::max<int64_t>(1, supers / (p.row_lanes * 4)));
  p.supers_per_split = ceil_div<int64_t>(supers, splits);
  p.splits = (int)ceil_div<int64_t>(supers, p.supers_per_split);
}

// `most_scratch`: bytes that the partial sums may take; a plan that needs more has fewer splits, down to the eight of a
// cluster, which needs none.
ColsPath cols_plan(int esize, int64_t A, int64_t B, int64_t C, size_t most_scratch, ColsPlan &p) {
  const int N = 16 / esize;
  // A thread per unit (a vector, or an element where rows are no whole vectors) walks over B rows, eight per round trip; eight
  // warps share them with the scalar kernel; super-rows start with more work per block and split further.  Measured on 446
  // shapes, us by a thread per unit / eight warps / super-rows: f32 [628, 2, 14604] 24 / 125 / 271, bf16 max [302, 4, 1280]
  // 3.0 / 8.3 / 10.0, f32 max [387, 73, 2325] 52 / 66 / 419; f16 max [5, 28, 88] 5.2 / 2.2 / 3.0, bf16 [358, 30691]
  // 17.2 / 14.4 / 19.2; f16 [34721, 1848] 3872 / 1921 / 22.
  const bool whole = C % N == 0;
  const int64_t units = whole ? A * C / N : A * C;
  if (whole ? B <= 8 || units >= 8LL * kNumSMs * B : B <= 16 || (B <= 32 && units >= 2048) || units >= 200 * B)
    return kDirect;
  if (C >= 32 && B <= (whole ? 32 : 64)) // with fewer columns most lanes of a warp would idle
    return kScalar;
  int64_t P = 1; // rows until the alignment repeats
  while (P * C % N != 0)
    P *= 2;
  const int64_t nvec = P * C / N;
  p = ColsPlan{};
  p.fold_rows = nvec <= 1024 && (P > 1 || nvec < kColsThreadsPerRow);
  if (p.fold_rows) {
    // as many rows as 256 threads hold, one vector each; a super-row of up to 1024 vectors takes 512 threads and two each
    p.P = P * std::max<int64_t>(1, std::min<int64_t>(kBlock / nvec, B / P));
    p.nvec = p.P * C / N;
    p.vpt = p.nvec <= kBlock ? 1 : 2;
    p.lpr = (int)ceil_div<int64_t>(p.nvec, p.vpt);
    p.row_lanes = (int)std::max<int64_t>(1, std::min<int64_t>(kBlock / p.lpr, B / p.P));
    p.threads = (int)ceil_div<int64_t>(p.lpr * p.row_lanes, 32) * 32;
    p.slabs = 1;
    split_cols(p, A, B);
  } else {
    // slabs of 32 vectors; every column's P partial sums go through the workspace, which is worth it while they are
    // few against the B rows
    if (P > 1 && (B < 16 * P || (B <= 512 && 2 * units >= kNumSMs * B)))
      return kScalar;
    p.P = P;
    p.nvec = nvec;
    p.vpt = 1;
    auto slabs_of = [&](int lpr) {
      p.lpr = lpr;
      p.row_lanes = kBlock / lpr;
      p.threads = kBlock;
      p.slabs = (int)ceil_div<int64_t>(nvec, lpr);
      split_cols(p, A, B);
    };
    int lpr = (int)std::min<int64_t>(kColsThreadsPerRow, pow2_ceil(nvec));
    if (g_cols_lpr_override > 0)
      lpr = std::min(lpr, g_cols_lpr_override);
    slabs_of(lpr);
    // narrower slabs (down to 128 bytes of a row) where they let eight blocks, a cluster, take all of B
    if (P == 1 && g_cols_lpr_override == 0)
      for (int w = lpr; p.splits > 8 && w >= 8; w /= 2) {
        ColsPlan wide = p;
        slabs_of(w);
        if (A * p.slabs * 8 >= 2 * kNumSMs || B <= 8LL * p.row_lanes * 16)
          p.splits = std::min(p.splits, 8), p.supers_per_split = ceil_div<int64_t>(B, p.splits);
        else
          p = wide;
      }
  }
  // One launch instead of two where at most eight blocks split the rows, or eight blocks need at most 16 loads per
  // thread (two latencies, less than the second launch).
  if (p.fold_rows && p.splits > 8 && std::max<int64_t>(1, B / p.P) <= 8LL * p.row_lanes * 16)
    p.splits = 8, p.supers_per_split = ceil_div<int64_t>(std::max<int64_t>(1, B / p.P), 8);
  const bool folds = p.fold_rows || p.P == 1; // a block's sums are one per column
  const int64_t fit = std::min<int64_t>(1 << 30, most_scratch / ((size_t)A * (folds ? 1 : p.P) * C * sizeof(float)));
  if (p.splits > (folds ? std::max<int64_t>(8, fit) : fit)) {
    if (!folds && fit < 1)
      return kScalar;
    const int64_t supers = std::max<int64_t>(1, B / p.P);
    p.supers_per_split = ceil_div<int64_t>(supers, folds && fit <= 8 ? 8 : fit);
    p.splits = (int)ceil_div<int64_t>(supers, p.supers_per_split);
  }
  p.cluster = p.splits > 1 && p.splits <= 8 && folds;
  return kSuper;
}

Plan make_plan(int esize, int64_t A, int64_t B, int64_t C, size_t most_scratch = SIZE_MAX) {
  Plan p{};
  const int N = 16 / esize;
  if (C == 1) {
    p.rows = true;
    const int64_t row_bytes = B * esize;
    const int64_t target_groups = 4LL * kNumSMs;
    p.segs = 1;
    p.seg_len = B;
    if (A < 2LL * kNumSMs && row_bytes > 32768) {
      // not more blocks than one wave holds, unless that leaves much of it empty
      int64_t segs = std::min<int64_t>(ceil_div<int64_t>(row_bytes, 16384),
                                       target_groups / A >= 3 ? target_groups / A : ceil_div<int64_t>(target_groups, A));
      int64_t seg_len = ceil_div<int64_t>(ceil_div<int64_t>(B, segs), N * 4) * (N * 4);
      segs = ceil_div<int64_t>(B, seg_len);
      p.segs = (int)segs;
      p.seg_len = seg_len;
    }
    const int64_t vec_per_seg = ceil_div<int64_t>(p.seg_len, N);
    p.tpr = (int)std::min<int64_t>(kBlock, pow2_ceil(ceil_div<int64_t>(vec_per_seg, 4)));
    if (p.segs > 1)
      p.tpr = kBlock;
    p.cluster = p.segs > 1 && p.segs <= 8;
    p.ws_bytes = p.declared_bytes = (p.segs > 1 && !p.cluster) ? (size_t)A * p.segs * sizeof(float) : 0;
  } else {
    p.rows = false;
    p.path = cols_plan(esize, A, B, C, most_scratch, p.cols);
    if (p.path == kSuper && (p.cols.splits > 1 || !(p.cols.fold_rows || p.cols.P == 1))) {
      p.declared_bytes = (size_t)p.cols.splits * A * (p.cols.fold_rows ? 1 : p.cols.P) * C * sizeof(float);
      p.ws_bytes = p.cols.cluster ? 0 : p.declared_bytes;
    }
  }
  return p;
}

template <typename T, int OP, typename OutT>
int launch(const T *in, OutT *out, int64_t A, int64_t B, int64_t C, void *ws,
           size_t ws_bytes, size_t most_scratch, cudaStream_t stream) {
  constexpr int N = 16 / sizeof(T);
  const Plan p = make_plan(sizeof(T), A, B, C, most_scratch);
  if (p.ws_bytes > 0 && (ws == nullptr || ws_bytes < p.ws_bytes))
    return B200_ERR_WORKSPACE;
  float *partial = static_cast<float *>(ws);
  if (p.rows) {
    const bool vec = aligned16(in) && (B % N == 0);
    const int tpr = vec ? p.tpr : std::max(p.tpr, 2 * N); // the edges of an unaligned row are one per thread
    const int groups_per_block = kBlock / tpr;
    const int64_t groups = A * p.segs;
    const int64_t grid = ceil_div<int64_t>(groups, groups_per_block);
    if (grid > 0x7fffffffLL)
      return B200_ERR_UNSUPPORTED;
    if (p.cluster) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3((unsigned)grid);
      cfg.blockDim = dim3(kBlock);
      cfg.stream = stream;
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = p.segs;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 2;
      cudaError_t e;
      if (vec)
        e = cudaLaunchKernelEx(&cfg, reduce_rows_kernel<T, OP, true, true, OutT>, in, out,
                               partial, A, B, tpr, p.segs, p.seg_len);
      else
        e = cudaLaunchKernelEx(&cfg, reduce_rows_kernel<T, OP, false, true, OutT>, in, out,
                               partial, A, B, tpr, p.segs, p.seg_len);
      return check_cuda(e);
    }
    if (!vec && B * (int64_t)sizeof(T) <= kChunkRow) {
      // 16 KB of rows per block, at most one per thread, fewer where that leaves SMs idle; the threads are dealt out evenly
      int64_t rows = std::min<int64_t>(kBlock, kChunkBytes / (B * (int64_t)sizeof(T)));
      rows = std::max<int64_t>(std::min<int64_t>(rows, 8), std::min<int64_t>(rows, ceil_div<int64_t>(A, 4 * kNumSMs)));
      int lanes = 1;
      while (lanes < 32 && 2 * lanes * rows <= kBlock)
        lanes *= 2;
      const int64_t blocks = ceil_div<int64_t>(A, rows);
      if (blocks <= 0x7fffffffLL)
        return launch_pdl(reduce_chunk_rows_kernel<T, OP, OutT>, dim3((unsigned)blocks), dim3(kBlock), 0, stream, in, out, A, (int)B,
                          lanes, (int)rows);
    }
    const int64_t nvec = B / N;
    if (p.segs == 1 && nvec <= 4LL * tpr) {
      const int vpt = (int)ceil_div<int64_t>(nvec, tpr);
      const int64_t row_blocks = ceil_div<int64_t>(A, groups_per_block);
      const unsigned pgrid = (unsigned)std::min<int64_t>(
          row_blocks, std::max<int64_t>(1, (int64_t)kNumSMs * g_rows_blocks_per_sm - g_reserved_blocks));
      auto go = [&](auto kernel) {
        return launch_pdl(kernel, dim3(pgrid), dim3(kBlock), 0, stream, in, out, A, B, tpr, g_prefetch_rows);
      };
      if (vpt <= 1)
        return vec ? go(reduce_short_rows_kernel<T, OP, 1, true, OutT>) : go(reduce_short_rows_kernel<T, OP, 1, false, OutT>);
      else if (vpt == 2)
        return vec ? go(reduce_short_rows_kernel<T, OP, 2, true, OutT>) : go(reduce_short_rows_kernel<T, OP, 2, false, OutT>);
      else
        return vec ? go(reduce_short_rows_kernel<T, OP, 4, true, OutT>) : go(reduce_short_rows_kernel<T, OP, 4, false, OutT>);
    }
    int rc;
    if (vec)
      rc = launch_pdl(reduce_rows_kernel<T, OP, true, false, OutT>, dim3((unsigned)grid), dim3(kBlock), 0, stream, in,
                      out, partial, A, B, tpr, p.segs, p.seg_len);
    else
      rc = launch_pdl(reduce_rows_kernel<T, OP, false, false, OutT>, dim3((unsigned)grid), dim3(kBlock), 0, stream, in,
                      out, partial, A, B, tpr, p.segs, p.seg_len);
    if (rc)
      return rc;
    if (p.segs > 1) {
      return launch_pdl(reduce_finalize_kernel<OP, OutT>, dim3((unsigned)ceil_div<int64_t>(A, 32)),
                        dim3(kFinalizeBlock), 0, stream, (const float *)partial, out, A, p.segs,
                        (int64_t)p.segs, (int64_t)1);
    }
    return B200_OK;
  }
  if (p.path == kDirect) {
    const bool vec = C % N == 0 && aligned16(in) && aligned16(out);
    const int64_t per_row = vec ? C / N : C, units = A * per_row, blocks = ceil_div<int64_t>(units, kBlock);
    if (blocks > 0x7fffffffLL)
      return B200_ERR_UNSUPPORTED;
    const FastDiv by_row((uint32_t)std::min<int64_t>(per_row, 0x7fffffff));
    if (vec)
      return launch_pdl(reduce_cols_direct_kernel<T, OP, true, OutT>, dim3((unsigned)blocks), dim3(kBlock), 0, stream, in, out, units, B,
                        C, per_row, by_row);
    return launch_pdl(reduce_cols_direct_kernel<T, OP, false, OutT>, dim3((unsigned)blocks), dim3(kBlock), 0, stream, in, out, units, B, C,
                      per_row, by_row);
  }
  if (p.path == kScalar) {
    const int64_t slabs = ceil_div<int64_t>(C, 32 * kScalarCols);
    if (A * slabs > 0x7fffffffLL)
      return B200_ERR_UNSUPPORTED;
    return launch_pdl(reduce_cols_scalar_kernel<T, OP, OutT>, dim3((unsigned)(A * slabs)), dim3(kBlock), 0, stream, in, out, A,
                      B, C, (int)slabs);
  }
  const ColsPlan &q = p.cols;
  const int64_t grid = A * q.slabs * q.splits;
  if (grid > 0x7fffffffLL)
    return B200_ERR_UNSUPPORTED;
  const size_t smem = (size_t)q.row_lanes * (q.fold_rows ? q.nvec : (int64_t)q.lpr * q.vpt) * N * sizeof(float);
  auto go = [&](auto kernel) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)q.threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = q.cluster ? q.splits : 1;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = q.cluster ? 2 : 1;
    return check_cuda(cudaLaunchKernelEx(&cfg, kernel, in, out, partial, A, B, C, q, g_prefetch_cols));
  };
  int rc;
  if (q.cluster)
    rc = q.vpt == 1 ? go(reduce_cols_kernel<T, OP, 1, true, OutT>) : go(reduce_cols_kernel<T, OP, 2, true, OutT>);
  else
    rc = q.vpt == 1 ? go(reduce_cols_kernel<T, OP, 1, false, OutT>) : go(reduce_cols_kernel<T, OP, 2, false, OutT>);
  if (rc || p.ws_bytes == 0)
    return rc;
  return launch_pdl(reduce_cols_fold_kernel<T, OP, OutT>, dim3((unsigned)ceil_div<int64_t>(A * C, 32)), dim3(kFinalizeBlock), 0,
                    stream, (const float *)partial, in, out, A, B, C, (int)(q.fold_rows ? 1 : q.P), q.splits, !q.fold_rows,
                    q.supers_per_split * q.P * C, q.P * C);
}

template <typename T>
int dispatch_op(int op, const void *in, void *out, int64_t A, int64_t B, int64_t C, void *ws,
                size_t ws_bytes, size_t most_scratch, cudaStream_t stream) {
  if (op == kSum)
    return launch<T, kSum, T>((const T *)in, (T *)out, A, B, C, ws, ws_bytes, most_scratch, stream);
  if (op == kMax)
    return launch<T, kMax, T>((const T *)in, (T *)out, A, B, C, ws, ws_bytes, most_scratch, stream);
  return B200_ERR_INVALID_ARG;
}

int esize_of(int dtype) {
  return dtype == B200_F32 ? 4 : (dtype == B200_F16 || dtype == B200_BF16) ? 2 : 0;
}

int reduce_within(int op, int dtype, const void *in, void *out, int64_t A, int64_t B, int64_t C, void *workspace,
                  size_t workspace_bytes, size_t most_scratch, cudaStream_t stream) {
  const int es = esize_of(dtype);
  if (!es || A < 0 || B < 0 || C < 0 || (op != kSum && op != kMax))
    return B200_ERR_INVALID_ARG;
  if (A == 0 && B == 0) { // nothing to reduce: a copy, as reduce_impl.h:70-73
    if (C == 0)
      return B200_OK;
    if (!in || !out)
      return B200_ERR_INVALID_ARG;
    return check_cuda(cudaMemcpyAsync(out, in, (size_t)C * es, cudaMemcpyDeviceToDevice, stream));
  }
  if (A == 0 || C == 0)
    return B200_OK; // empty output
  if (B == 0 || !in || !out)
    return B200_ERR_INVALID_ARG;
  switch (dtype) {
  case B200_F32:
    return dispatch_op<float>(op, in, out, A, B, C, workspace, workspace_bytes, most_scratch, stream);
  case B200_F16:
    return dispatch_op<__half>(op, in, out, A, B, C, workspace, workspace_bytes, most_scratch, stream);
  default:
    return dispatch_op<__nv_bfloat16>(op, in, out, A, B, C, workspace, workspace_bytes, most_scratch, stream);
  }
}

// The partial sums of a column reduction that splits B over one wave of blocks, each 32 vectors of a row (32 elements, if
// a row is no whole number of vectors) wide: what b200_reduce_no_alloc measures shapes by.
size_t plain_split_bytes(int esize, int64_t A, int64_t B, int64_t C) {
  const int64_t units = C % (16 / esize) == 0 ? C / (16 / esize) : C;
  const int64_t width = std::min<int64_t>(kColsThreadsPerRow, pow2_ceil(units)), blocks = A * ceil_div<int64_t>(units, width);
  int64_t splits = std::min<int64_t>(ceil_div<int64_t>(4 * kNumSMs, blocks), std::max<int64_t>(1, B / (kBlock / width * 4)));
  splits = ceil_div<int64_t>(B, ceil_div<int64_t>(B, splits));
  return splits > 1 ? (size_t)splits * A * C * sizeof(float) : 0;
}

} // namespace
} // namespace b200

using namespace b200;

// Measurement hook (not part of the drop-in ABI): pins the column plan's threads per slab row
// (0 = the shape rule).  Workspace sizes follow the pinned plan, so ask for them after calling this.
extern "C" void b200_reduce_cols_plan_override(int threads_per_row) { g_cols_lpr_override = threads_per_row; }

extern "C" void b200_reduce_reserve_blocks(int blocks) { g_reserved_blocks = blocks > 0 ? blocks : 0; }

extern "C" void b200_reduce_tune(int prefetch_cols, int prefetch_rows, int cols_blocks_per_sm, int rows_blocks_per_sm) {
  g_prefetch_cols = prefetch_cols;
  g_prefetch_rows = prefetch_rows;
  g_cols_blocks_per_sm = cols_blocks_per_sm > 0 ? cols_blocks_per_sm : 4;
  g_rows_blocks_per_sm = rows_blocks_per_sm > 0 ? rows_blocks_per_sm : 4;
}

extern "C" size_t b200_reduce_workspace_bytes(int op, int dtype, int64_t A, int64_t B, int64_t C) {
  (void)op;
  const int es = esize_of(dtype);
  if (!es || A <= 0 || B <= 0 || C <= 0)
    return 0;
  return make_plan(es, A, B, C).declared_bytes;
}

// What a call really uses: 0 where the blocks that split B fold through distributed shared memory, for which
// b200_reduce_workspace_bytes names the size of their partial sums all the same (its answer is older than that fold,
// and callers size fixed buffers by it).  For callers that allocate on every call.
extern "C" size_t b200_reduce_scratch_bytes(int op, int dtype, int64_t A, int64_t B, int64_t C) {
  (void)op;
  const int es = esize_of(dtype);
  if (!es || A <= 0 || B <= 0 || C <= 0)
    return 0;
  return make_plan(es, A, B, C).ws_bytes;
}

extern "C" int b200_reduce(int op, int dtype, const void *in, void *out, int64_t A, int64_t B,
                           int64_t C, void *workspace, size_t workspace_bytes,
                           cudaStream_t stream) {
  return reduce_within(op, dtype, in, out, A, B, C, workspace, workspace_bytes, SIZE_MAX, stream);
}

extern "C" int b200_reduce_sum_to_f32(int dtype, const void *in, float *out, int64_t A, int64_t B,
                                      int64_t C, void *workspace, size_t workspace_bytes,
                                      cudaStream_t stream) {
  const int es = esize_of(dtype);
  if (!es || A <= 0 || B <= 0 || C <= 0 || !in || !out)
    return B200_ERR_INVALID_ARG;
  switch (dtype) {
  case B200_F32:
    return launch<float, kSum, float>((const float *)in, out, A, B, C, workspace, workspace_bytes, SIZE_MAX, stream);
  case B200_F16:
    return launch<__half, kSum, float>((const __half *)in, out, A, B, C, workspace, workspace_bytes, SIZE_MAX, stream);
  default:
    return launch<__nv_bfloat16, kSum, float>((const __nv_bfloat16 *)in, out, A, B, C, workspace,
                                              workspace_bytes, SIZE_MAX, stream);
  }
}

extern "C" int b200_cast_from_f32(int dtype, const float *in, void *out, int64_t n,
                                  cudaStream_t stream) {
  if (n < 0 || !esize_of(dtype))
    return B200_ERR_INVALID_ARG;
  if (n == 0)
    return B200_OK;
  if (!in || !out)
    return B200_ERR_INVALID_ARG;
  const unsigned grid = (unsigned)ceil_div<int64_t>(n, kBlock);
  switch (dtype) {
  case B200_F32:
    cast_from_f32_kernel<float><<<grid, kBlock, 0, stream>>>(in, (float *)out, n);
    break;
  case B200_F16:
    cast_from_f32_kernel<__half><<<grid, kBlock, 0, stream>>>(in, (__half *)out, n);
    break;
  default:
    cast_from_f32_kernel<__nv_bfloat16><<<grid, kBlock, 0, stream>>>(in, (__nv_bfloat16 *)out, n);
  }
  return check_launch();
}

// ---- reduction without a caller-provided workspace ----------------------------
// Scratch for b200_reduce_no_alloc: one fixed block of device memory per GPU that
// loads this library, held until the process exits.
namespace {
constexpr size_t kStaticScratchBytes = 1u << 20;
static __device__ __align__(256) unsigned char g_reduce_static_scratch[kStaticScratchBytes];

// `g_reduce_static_scratch` names a host-side handle here, not device memory: the
// device address has to be asked for, once per device, with that device current.
int static_scratch_for_current_device(void **ptr) {
  constexpr int kMaxDevices = 64;
  static std::mutex mu;
  static void *addr[kMaxDevices] = {};
  int dev = 0;
  if (int rc = check_cuda(cudaGetDevice(&dev)))
    return rc;
  if (dev < 0 || dev >= kMaxDevices)
    return B200_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    void *p = nullptr;
    if (int rc = check_cuda(cudaGetSymbolAddress(&p, g_reduce_static_scratch)))
      return rc;
    addr[dev] = p;
  }
  *ptr = addr[dev];
  return B200_OK;
}
} // namespace

extern "C" size_t b200_reduce_no_alloc_max_bytes(void) { return kStaticScratchBytes; }

// Takes what fits by either measure: the plan's own scratch or that of a plain split, and makes a plan that fits.
extern "C" int b200_reduce_no_alloc(int op, int dtype, const void *in, void *out, int64_t A, int64_t B,
                                    int64_t C, cudaStream_t stream) {
  const int es = esize_of(dtype);
  size_t need = 0;
  if (es && A > 0 && B > 0 && C > 0) {
    if (b200_reduce_workspace_bytes(op, dtype, A, B, C) > kStaticScratchBytes &&
        (C == 1 || plain_split_bytes(es, A, B, C) > kStaticScratchBytes))
      return B200_ERR_WORKSPACE;
    need = make_plan(es, A, B, C, kStaticScratchBytes).ws_bytes;
  }
  void *scratch = nullptr;
  if (need > 0)
    if (int rc = static_scratch_for_current_device(&scratch))
      return rc;
  return reduce_within(op, dtype, in, out, A, B, C, scratch, need ? kStaticScratchBytes : 0, kStaticScratchBytes, stream);
}
