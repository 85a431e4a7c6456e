// dist.cu - distance (non-equi) join: all pairs of R and S points within a radius.
//
// Reference: the 2-D GPU join joins/blockJoin_gpu/complex_block/dire_join
// (eval, count and join kernels, join_gpu.cu:12-130; VAL_NUM 2, tuple.h:18-30)
// and the CPU joins joins/CPU_JOIN/3d_cpu/nestLoopJoin.cc (eval :73-84, loop
// :86-101; VAL_NUM 3) and joins/blockJoin_gpu/complex_block/2d_cpu.  A left
// point l (from S) and a right point r (from R) match when, in IEEE double with
// every operation rounded on its own,
//   temp = 0; for each dimension i: t = r.val[i] - l.val[i]; temp += t * t;
//   temp < radius * radius                   (radius = DISTANCE = 1 there).
//
// Grid.  A match has |r.val[i] - l.val[i]| < rho = |radius| in exact arithmetic
// in every dimension: rounding is monotone, so a difference of rho or more
// rounds to rho or more, its square to radius^2 or more, and the other squares
// only add.  So R is grouped by cells of width 2 rho (hashed over all
// dimensions into 2 to 4 buckets per point) and an S point looks only at the
// cells that hold [l - rho, l + rho], two per dimension on average: a few
// lookups and a few candidates per S point instead of |R| compares.  The cell
// number is a monotone function of the coordinate (dist_cell), so the cells
// from that of l - rho (rounded down) to that of l + rho (rounded up) hold
// every match whatever the rounding; a width fixed by the radius keeps the
// cells small when a few points lie far out.  Points with a NaN or an infinite
// coordinate match nothing (NaN and inf - inf differences are NaN, the others
// infinite, and neither is below any radius^2) and are left out; radius^2 of
// zero or NaN matches nothing at all.
//
// Candidates.  The grouped R keeps one 16-byte entry per point, its
// coordinates rounded to float and its row.  A candidate is dropped when its
// float distance is past a bound that no match reaches (dist_screen_bound);
// the others get the reference's predicate on the doubles (__dsub_rn,
// __dmul_rn, __dadd_rn in its order: no fused multiply-add), so the matches
// are the reference's, bit for bit.  FP64 runs at 1/64 of the FP32 rate here
// (a warp instruction takes 16 cycles, however few lanes are active), so the
// candidates that pass the screen are collected and tested by full warps: at
// once, most steps of a probe warp would take the double path for one or two
// lanes.  Two of an S point's cells may share a bucket (when its reach spans
// three cells somewhere), which is then looked at once: every R point lies in one
// bucket, so no pair comes twice.
//
// Launches: cells (histogram with the points' ranks in their buckets), scan,
// placement, probe, and where buckets are crowded one more for these (below); few
// S points: one launch, no grid.  A probe warp takes 32 S points: each lane finds its point's
// cells, then groups of 4 (2-D) or 8 (3-D) lanes share a point, a lane per cell,
// and walk the buckets together, two candidates a step; the pairs that pass
// the screen collect in shared memory, and full buffers are tested and become
// rows with one atomic add on the cursor and coalesced 8-byte stores (the row
// order is not deterministic, the row multiset is).  Count-only mode sums
// per-thread counters.
// Both calls of a join (count, then rows): 2^19 x 2^19 2-D points far apart by
// all pairs 37.7 ms, by the grid with a lane per S point and the predicate in
// the step 0.356 ms, here 0.237 (the probe 87 -> 46 us; 50 when the buckets of a
// point's cells were unrelated and had to be compared); 100 003 x 150 001 points
// of a 3-D box with about three matches each 77.7, 1.04 and 0.221 ms (the probe
// 430 -> 53 us).  Bound by the chain of dependent loads and shuffles per S point
// (half of the warps resident, the issue slots 30% busy).
#include <float.h>
#include <math.h>

#include <algorithm>
#include <functional>

#include "ej_device.cuh"
#include "ej_entry.h"

namespace {

constexpr int DJ_THREADS = 256;
constexpr int DJ_WARPS = DJ_THREADS / 32;
constexpr int DJ_BUF = 192;  // candidate pairs a warp collects (tested past 128; a step adds at most 64)
// points per launch sequence: 32-bit rows in the grid's entries, and at most 2.5 GB
// of scratch for the grid, 0.25 GB for crowded buckets; larger relations go in pieces
constexpr uint64_t DJ_RPIECE = 1ull << 26;
constexpr uint64_t DJ_SPIECE = 1ull << 26;
constexpr uint64_t DJ_LEAST_PIECE = 1ull << 16;  // R pieces get no smaller when memory is short
constexpr uint64_t DJ_FEW_RPIECE = 1ull << 31;  // without a grid

template <int D>
struct Point {
  int32_t id;
  double val[D];
};
static_assert(sizeof(Point<2>) == sizeof(ej_point2) && sizeof(Point<3>) == sizeof(ej_point3), "point layouts");

// the handle's words of the list of crowded buckets (DistCrowd::header), behind the row cursor
constexpr int DJ_CROWD_WORD = 1;

// the radius as the kernels use it
struct DistRadius {
  double rho;    // |radius|
  double inv_w;  // 1 / (2 rho): cells of width 2 rho; 0 (one cell) when that is infinite
  double r2;     // radius^2, rounded as the reference's
  float rho_up;  // rho rounded up to float
};

template <int D>
__device__ __forceinline__ bool dist_finite(const Point<D>& p) {
  bool ok = true;
#pragma unroll
  for (int i = 0; i < D; i++)
    ok = ok && ((unsigned long long)__double_as_longlong(p.val[i]) & 0x7FF0000000000000ull) != 0x7FF0000000000000ull;
  return ok;
}

// The cell number of a finite coordinate: floor(x inv_w) up to 2^50 cells from
// the origin; past that, where neighbouring doubles are rho / 4 or more
// apart, every representable x inv_w is a cell of its own, numbered on by its
// bit pattern.  Monotone in x throughout (the product is rounded monotonely),
// and [l - rho, l + rho] spans at most 3 cells in the first range, 12 in the
// second.
// (The magnitude test is on the exponent bits, off the FP64 pipe.)
__device__ __forceinline__ long long dist_cell(double x, double inv_w) {
  const double t = __dmul_rn(x, inv_w);  // x finite: inv_w = 0 gives 0
  const unsigned long long mag = (unsigned long long)__double_as_longlong(t) & 0x7FFFFFFFFFFFFFFFull;
  constexpr unsigned long long FAR = 0x4310000000000000ull;  // the bits of 2^50
  if (mag < FAR) return __double2ll_rd(t);
  const long long c = (long long)((1ull << 50) + (mag - FAR));
  return __double_as_longlong(t) < 0 ? -c : c;
}

// a bound of [l - rho, l + rho] kept finite (R's points are)
__device__ __forceinline__ double dist_clamp(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b & 0x7FFFFFFFFFFFFFFFull) == 0x7FF0000000000000ull ? __longlong_as_double((long long)(b - 1)) : x;
}

// the bucket of a cell: the cells of a block of two per dimension are neighbours,
// told by their numbers' lowest bits, and a multiplicative hash places the block.
// So the 2^D cells of a point whose reach spans two per dimension never share a
// bucket, and most of them lie next to each other.
template <int D>
__device__ __forceinline__ uint32_t dist_bucket(const long long (&c)[D], uint32_t bits) {
  unsigned long long x = (unsigned long long)(c[0] >> 1) * 0x9E3779B97F4A7C15ull;
  uint32_t low = (uint32_t)c[0] & 1u;
#pragma unroll
  for (int i = 1; i < D; i++) {
    x ^= x >> 32;
    x = (x + (unsigned long long)(c[i] >> 1)) * 0xD1342543DE82EF95ull;
    low |= ((uint32_t)c[i] & 1u) << i;
  }
  x ^= x >> 32;
  x *= 0x9E3779B97F4A7C15ull;
  return (uint32_t)(x >> (64u - (bits - D))) << D | low;
}

// a / n; cells span one or two per dimension nearly always
__device__ __forceinline__ uint32_t dist_div(uint32_t a, uint32_t n) { return n <= 2u ? a >> (n - 1u) : a / n; }

// the reference's predicate, operation by operation
template <int D>
__device__ __forceinline__ bool dist_match(const Point<D>& r, const Point<D>& l, double r2) {
  double temp = 0.0;
#pragma unroll
  for (int i = 0; i < D; i++) {
    const double t = __dsub_rn(r.val[i], l.val[i]);
    temp = __dadd_rn(temp, __dmul_rn(t, t));
  }
  return temp < r2;
}

// Bound of the float screen: a pair whose float squared distance is above it
// is no match.  For a match, with l at most m away from the origin in every
// dimension and rho the radius, r in a looked-at cell is at most m + 4 rho away;
// rounding both to float moves each difference by at most
// e = 2^-24 (2 m + 4 rho) (and 2^-149 twice below the normal range), so the
// float distance is at most (rho + sqrt(3) e) times 1 + 2^-18, which also
// covers the rounding of the float operations, the squares' underflow
// (2^-140) and the predicate's own rounding.  Past 10^18 the squares could
// overflow: no screen (infinity; NaN distances pass it too).
__device__ __forceinline__ float dist_screen_bound(float rho_up, float m) {
  if (!(m < 1e18f) || !(rho_up < 1e18f)) return INFINITY;
  const float e = __fadd_ru(__fmul_ru(0x1p-24f, __fadd_ru(__fmul_ru(2.0f, m), __fmul_ru(4.0f, rho_up))), 0x1p-140f);
  const float b = __fmul_ru(__fadd_ru(rho_up, __fmul_ru(1.7320509f, e)), 1.0f + 0x1p-18f);
  return __fadd_ru(__fmul_ru(__fmul_ru(b, b), 1.0f + 0x1p-18f), 0x1p-140f);
}

// an S point as the screen uses it: its coordinates as floats, and the bound
template <int D>
__device__ __forceinline__ float dist_screen_point(const double (&v)[D], float rho_up, float (&x)[D]) {
  float m = 0.0f;
#pragma unroll
  for (int d = 0; d < D; d++) {
    x[d] = __double2float_rn(v[d]);
    m = fmaxf(m, __fmul_ru(fabsf(x[d]), 1.0f + 0x1p-23f));
  }
  return dist_screen_bound(rho_up, m);
}

template <int D>
struct RowOf;
template <>
struct RowOf<2> {
  using type = ej_point_result2;
};
template <>
struct RowOf<3> {
  using type = ej_point_result3;
};

// A warp's lanes whose bucket is the same take consecutive ranks with one
// atomic: a bucket that holds most of R costs 1/32 of the atomics.
template <int D>
__global__ void __launch_bounds__(256)
dist_cell_kernel(const Point<D>* __restrict__ R, uint32_t nR, DistRadius rad, uint32_t bits,
                 uint32_t* __restrict__ count, uint2* __restrict__ place) {
  const uint32_t lane = threadIdx.x & 31u;
  for (uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~31ull; w < nR;
       w += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t i = w + lane;
    uint32_t b = 0xFFFFFFFFu;  // past nR, or a point that matches nothing
    if (i < nR) {
      const Point<D> p = R[i];
      if (dist_finite<D>(p)) {
        long long c[D];
#pragma unroll
        for (int d = 0; d < D; d++) c[d] = dist_cell(p.val[d], rad.inv_w);
        b = dist_bucket<D>(c, bits);
      }
    }
    const unsigned peers = __match_any_sync(EJ_FULL_MASK, b);
    const int leader = __ffs(peers) - 1;
    uint32_t first = 0;
    if ((int)lane == leader && b != 0xFFFFFFFFu) first = atomicAdd(count + b, (uint32_t)__popc(peers));
    first = __shfl_sync(EJ_FULL_MASK, first, leader);
    if (i < nR) place[i] = make_uint2(b, first + __popc(peers & ej_lanemask_lt()));
  }
}

template <int D>
__global__ void __launch_bounds__(256)
dist_place_kernel(const Point<D>* __restrict__ R, uint32_t nR, const uint2* __restrict__ place,
                  const uint32_t* __restrict__ start, float4* __restrict__ grid) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nR; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint2 pl = place[i];
    if (pl.x == 0xFFFFFFFFu) continue;
    const Point<D> p = R[i];
    float4 e;
    e.x = __double2float_rn(p.val[0]);
    e.y = __double2float_rn(p.val[1]);
    e.z = D == 3 ? __double2float_rn(p.val[D - 1]) : 0.0f;
    e.w = __uint_as_float((uint32_t)i);
    grid[start[pl.x] + pl.y] = e;
  }
}

// Tests the n candidate pairs {S row, R row} of a warp's buffer and writes the
// matches as result rows, laid out as the reference's (padding zero): dims 2
// {lid, lval[2], rid, rval[2]}, dims 3 {lval[3], rval[3], lid, rid}; consecutive
// lanes write consecutive 8-byte words.  Count-only: returns the lane's matches.
template <int D, bool COUNT_ONLY>
__device__ __forceinline__ uint32_t dist_flush(uint2* buf, uint32_t n, const Point<D>* __restrict__ R,
                                               const Point<D>* __restrict__ S, double r2,
                                               typename RowOf<D>::type* __restrict__ out, uint64_t cap,
                                               unsigned long long* cursor) {
  constexpr uint32_t WORDS = sizeof(typename RowOf<D>::type) / 8;
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t rows = 0;
  __syncwarp();
  for (uint32_t k0 = 0; k0 < n; k0 += 32) {
    uint2 pr = make_uint2(0u, 0u);
    bool hit = false;
    if (k0 + lane < n) {
      pr = buf[k0 + lane];
      hit = dist_match<D>(R[pr.y], S[pr.x], r2);
    }
    if (COUNT_ONLY) {
      rows += hit ? 1u : 0u;
      continue;
    }
    // the matches move to the front, behind those of the steps before (all
    // lanes have read their pairs of this step)
    const unsigned hits = __ballot_sync(EJ_FULL_MASK, hit);
    if (hit) buf[rows + __popc(hits & ej_lanemask_lt())] = pr;
    rows += __popc(hits);
    __syncwarp();
  }
  if (COUNT_ONLY || rows == 0) return rows;
  unsigned long long off = 0;
  if (lane == 0) off = atomicAdd(cursor, (unsigned long long)rows);
  off = __shfl_sync(EJ_FULL_MASK, off, 0);
  for (uint32_t k = lane; k < rows * WORDS; k += 32) {
    const uint32_t row = k / WORDS, word = k - row * WORDS;
    if (off + row >= cap) break;
    const uint2 pr = buf[row];
    const Point<D>& l = S[pr.x];
    const Point<D>& r = R[pr.y];
    unsigned long long v;
    if (D == 2) {
      const Point<D>& p = word < 3 ? l : r;
      const uint32_t q = word < 3 ? word : word - 3;
      v = q == 0 ? (unsigned long long)(uint32_t)p.id : (unsigned long long)__double_as_longlong(p.val[q - 1]);
    } else {
      v = word == 6 ? (unsigned long long)(uint32_t)l.id | (unsigned long long)(uint32_t)r.id << 32
                    : (unsigned long long)__double_as_longlong(word < 3 ? l.val[word] : r.val[word - 3]);
    }
    reinterpret_cast<unsigned long long*>(out + off)[k] = v;
  }
  __syncwarp();
  return rows;
}

// ---- crowded buckets -------------------------------------------------------------
// A bucket of DJ_CROWD rows or more (a radius that reaches many points, points in
// few cells) would be walked by one lane per S point and cell, and few S points by
// few warps.  Its lookups become items of a list, {first S row, owners, first grid
// entry, end}, instead: the owners (bits) are those of the probe warp's 32 S points
// that look at it, the entries a part of the bucket.  A kernel of its own takes the
// items, a warp each, all lanes at work: k owners and 32 / k entries a step.
// The list has two parts: buckets in parts, as many as fill the device when few S
// points are concerned, and whole buckets, once the first part is full.  What finds
// no room there either (many S points in many crowded buckets) is walked as the
// others are, by then with most lanes at work.
// Counts of 2^20 R and 64 to 1500 S points, a radius that reaches 0.3% of R: walked
// 4.9 to 4.5 ms; 2^24 R and 400 S points 121 ms walked, 1.7 listed.
constexpr uint32_t DJ_CROWD = 256;
constexpr uint32_t DJ_ITEM_ROWS = 1024;     // least entries of a part
constexpr uint32_t DJ_SPLIT = 1u << 18;     // items in parts
constexpr uint64_t DJ_WHOLE = 1u << 14;     // whole buckets: 8 per 32 S points, at least these

struct DistCrowd {
  uint4* items;      // [DJ_SPLIT + whole]
  uint32_t* header;  // items {in parts, whole}, counted on past the room; {taken}
  uint32_t whole;
  uint32_t parts;  // parts of a bucket at most
};

// The matches of the item's owners among its entries: candidates collect in buf
// (held of them), full buffers are tested.  Count-only: returns the lane's matches
// among those tested.
template <int D, bool COUNT_ONLY>
__device__ __forceinline__ uint32_t dist_crowd(const uint4& it, const Point<D>* __restrict__ R,
                                               const Point<D>* __restrict__ S, const float4* __restrict__ grid,
                                               const DistRadius& rad, typename RowOf<D>::type* __restrict__ out,
                                               uint64_t cap, unsigned long long* cursor, uint2* buf, uint32_t& held) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t lg = 0;  // 2^lg owners a step
  while ((1u << lg) < (uint32_t)__popc(it.y)) lg++;
  uint32_t m = it.y;
  for (uint32_t i = lane & ((1u << lg) - 1u); i; i--) m &= m - 1u;
  const bool ok = m != 0u;
  const uint32_t si = it.x + (ok ? __ffs(m) - 1u : 0u);
  float x[D], bound;
  {
    double v[D];
#pragma unroll
    for (int d = 0; d < D; d++) v[d] = ok ? S[si].val[d] : 0.0;
    bound = dist_screen_point<D>(v, rad.rho_up, x);
  }
  uint32_t rows = 0;
  constexpr int U = 4;
  for (uint32_t q = it.z; q < it.w; q += U * (32u >> lg)) {
    float4 e[U];
    bool pass[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint32_t at = q + u * (32u >> lg) + (lane >> lg);
      pass[u] = ok && at < it.w;
      e[u] = pass[u] ? __ldg(grid + at) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    bool some = false;
#pragma unroll
    for (int u = 0; u < U; u++) {
      const float dx = e[u].x - x[0], dy = e[u].y - x[1], dz = D == 3 ? e[u].z - x[D - 1] : 0.0f;
      pass[u] = pass[u] && !(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > bound);
      some |= pass[u];
    }
    if (!__any_sync(EJ_FULL_MASK, some)) continue;
#pragma unroll
    for (int u = 0; u < U; u++) {
      const unsigned b = __ballot_sync(EJ_FULL_MASK, pass[u]);
      if (pass[u]) buf[held + __popc(b & ej_lanemask_lt())] = make_uint2(si, __float_as_uint(e[u].w));
      held += __popc(b);
      if (held > DJ_BUF - 64) {
        const uint32_t n = dist_flush<D, COUNT_ONLY>(buf, held, R, S, rad.r2, out, cap, cursor);
        if (COUNT_ONLY) rows += n;
        held = 0;
      }
    }
  }
  return rows;
}

// Lists the entries [from, end) of a crowded bucket for those of the warp's S points
// (the first is s0) that look at it; false: no room.
__device__ __forceinline__ bool dist_list(const DistCrowd& crowd, uint32_t s0, uint32_t owners, uint32_t from,
                                          uint32_t end) {
  const uint32_t lane = threadIdx.x & 31u, len = end - from;
  const uint32_t want = min(len / DJ_ITEM_ROWS + 1u, crowd.parts);
  const uint32_t step = (len + want - 1u) / want, parts = (len + step - 1u) / step;
  volatile const uint32_t* listed = crowd.header;  // (looked at first, so that the counters stay small)
  uint32_t at = DJ_SPLIT, whole = crowd.whole;
  if (lane == 0) {
    if (listed[0] < DJ_SPLIT) at = atomicAdd(crowd.header, parts);
    if (at + parts > DJ_SPLIT && listed[1] < crowd.whole) whole = atomicAdd(crowd.header + 1, 1u);
  }
  at = __shfl_sync(EJ_FULL_MASK, at, 0);
  whole = __shfl_sync(EJ_FULL_MASK, whole, 0);
  const bool fits = at + parts <= DJ_SPLIT;
  for (uint32_t j = lane; j < parts && at + j < DJ_SPLIT; j += 32) {  // (empty items at the first part's end)
    const uint32_t q = from + j * step;
    crowd.items[at + j] = fits ? make_uint4(s0, owners, q, min(q + step, end)) : make_uint4(0u, 0u, 0u, 0u);
  }
  if (fits) return true;
  if (whole >= crowd.whole) return false;
  if (lane == 0) crowd.items[DJ_SPLIT + whole] = make_uint4(s0, owners, from, end);
  return true;
}

// the listed items, a warp each until none is left
template <int D, bool COUNT_ONLY>
__global__ void __launch_bounds__(DJ_THREADS)
dist_crowd_kernel(const Point<D>* __restrict__ R, const Point<D>* __restrict__ S, const float4* __restrict__ grid,
                  DistCrowd crowd, DistRadius rad, typename RowOf<D>::type* __restrict__ out, uint64_t cap,
                  unsigned long long* cursor) {
  const uint32_t split = min(crowd.header[0], DJ_SPLIT), n = split + min(crowd.header[1], crowd.whole);
  if (n == 0) return;
  __shared__ uint2 bufs[DJ_WARPS][DJ_BUF];
  __shared__ unsigned long long warp_tmp[DJ_WARPS + 1];
  uint2* buf = bufs[threadIdx.x >> 5];
  uint32_t held = 0;
  unsigned long long local = 0;
  for (;;) {
    uint32_t i = 0;
    if ((threadIdx.x & 31u) == 0) i = atomicAdd(crowd.header + 2, 1u);
    i = __shfl_sync(EJ_FULL_MASK, i, 0);
    if (i >= n) break;
    local += dist_crowd<D, COUNT_ONLY>(__ldg(crowd.items + (i < split ? i : DJ_SPLIT + (i - split))), R, S, grid, rad, out, cap, cursor, buf, held);
  }
  if (held) {
    const uint32_t rows = dist_flush<D, COUNT_ONLY>(buf, held, R, S, rad.r2, out, cap, cursor);
    if (COUNT_ONLY) local += rows;
  }
  if (COUNT_ONLY) {
    unsigned long long total;
    ej_block_exclusive_sum<DJ_THREADS, unsigned long long>(local, warp_tmp, &total);
    if (threadIdx.x == 0 && total) atomicAdd(cursor, total);
  }
}

template <int D, bool COUNT_ONLY>
__global__ void __launch_bounds__(DJ_THREADS, 4)
dist_probe_kernel(const Point<D>* __restrict__ R, const Point<D>* __restrict__ S, uint32_t nS,
                  const uint32_t* __restrict__ start, const float4* __restrict__ grid, uint32_t bits, DistRadius rad,
                  DistCrowd crowd, typename RowOf<D>::type* __restrict__ out, uint64_t cap,
                  unsigned long long* cursor) {
  constexpr int G = D == 2 ? 4 : 8;  // lanes of an S point: its cells, when no dimension has three
  __shared__ uint2 bufs[DJ_WARPS][DJ_BUF];
  __shared__ unsigned long long warp_tmp[DJ_WARPS + 1];
  const uint32_t lane = threadIdx.x & 31u, g = lane % G;
  const unsigned group = (D == 2 ? 0xFu : 0xFFu) << (lane - g);  // the lanes of this lane's S point
  uint2* buf = bufs[threadIdx.x >> 5];
  uint32_t held = 0;  // pairs in the warp's buffer
  unsigned long long local = 0;
  for (uint64_t w = ((uint64_t)blockIdx.x * DJ_THREADS + threadIdx.x) & ~31ull; w < nS;
       w += (uint64_t)gridDim.x * DJ_THREADS) {
    // the lane's own S point: the first of the cells that hold [l - rho, l +
    // rho] and their number in every dimension (at most 12)
    long long lo[D];
    uint32_t spans = 0;  // 8 bits per dimension; 0: no point
    float x[D], bound;
    {
      const uint64_t si = w + lane;
      Point<D> l;
      bool ok = si < nS;
      if (ok) {
        l = S[si];
        ok = dist_finite<D>(l);
      }
      double v[D];
#pragma unroll
      for (int d = 0; d < D; d++) {
        v[d] = ok ? l.val[d] : 0.0;
        lo[d] = dist_cell(dist_clamp(__dsub_rd(v[d], rad.rho)), rad.inv_w);
        const uint32_t span = (uint32_t)(dist_cell(dist_clamp(__dadd_ru(v[d], rad.rho)), rad.inv_w) - lo[d]) + 1u;
        spans |= (ok ? span : 0u) << (8 * d);
      }
      bound = dist_screen_point<D>(v, rad.rho_up, x);
    }
    // 32 / G of the warp's S points at a time, G lanes each
    for (int t = 0; t < G; t++) {
      const int owner = t * (32 / G) + (int)(lane / G);
      long long c0[D];
      float xs[D];
#pragma unroll
      for (int d = 0; d < D; d++) {
        c0[d] = __shfl_sync(EJ_FULL_MASK, lo[d], owner);
        xs[d] = __shfl_sync(EJ_FULL_MASK, x[d], owner);
      }
      const uint32_t sp = __shfl_sync(EJ_FULL_MASK, spans, owner);
      const float bd = __shfl_sync(EJ_FULL_MASK, bound, owner);
      const uint32_t n0 = sp & 0xFFu, n1 = sp >> 8 & 0xFFu, n2 = D == 3 ? sp >> 16 : 1u;
      const uint32_t cells = n0 * n1 * n2;
      for (uint32_t first = 0; __any_sync(EJ_FULL_MASK, first < cells); first += G) {
        const uint32_t k = first + g;
        uint32_t p = 0, end = 0, b = 0xFFFFFFFFu;
        if (k < cells) {
          const uint32_t k1 = dist_div(k, n0);
          long long c[D];
          c[0] = c0[0] + (k - k1 * n0);
          const uint32_t k2 = dist_div(k1, n1);
          c[1] = c0[1] + (k1 - k2 * n1);
          if (D == 3) c[D - 1] = c0[D - 1] + k2;
          b = dist_bucket<D>(c, bits);
          // the point's earlier cells in this bucket, which only points whose
          // reach spans three cells or more somewhere can have: in this round of
          // G cells (below), and in the rounds before
          for (uint32_t e = 0; e < first; e++) {
            const uint32_t e1 = e / n0, e2 = e1 / n1;
            long long f[D];
            f[0] = c0[0] + (e - e1 * n0);
            f[1] = c0[1] + (e1 - e2 * n1);
            if (D == 3) f[D - 1] = c0[D - 1] + e2;
            if (dist_bucket<D>(f, bits) == b) b = 0xFFFFFFFFu;
          }
        }
        unsigned same = 0;
        if (__any_sync(EJ_FULL_MASK, n0 > 2u || n1 > 2u || n2 > 2u))
          same = __match_any_sync(EJ_FULL_MASK, b) & group & ej_lanemask_lt();
        if (b != 0xFFFFFFFFu && same == 0) {
          p = __ldg(start + b);
          end = __ldg(start + b + 1);
        }
        uint32_t longest = __reduce_max_sync(EJ_FULL_MASK, end - p);
        if (longest >= DJ_CROWD) {
          for (unsigned many = __ballot_sync(EJ_FULL_MASK, end - p >= DJ_CROWD); many;) {
            const int leader = __ffs(many) - 1;
            const uint32_t q = __shfl_sync(EJ_FULL_MASK, p, leader), qe = __shfl_sync(EJ_FULL_MASK, end, leader);
            const bool here = (many >> lane & 1u) && p == q;
            many &= ~__ballot_sync(EJ_FULL_MASK, here);
            const uint32_t owners = __reduce_or_sync(EJ_FULL_MASK, here ? 1u << owner : 0u);
            if (dist_list(crowd, (uint32_t)w, owners, q, qe) && here) p = end;
          }
          longest = __reduce_max_sync(EJ_FULL_MASK, end - p);
        }
        for (uint32_t k2 = 0; k2 < longest; k2 += 2) {
          bool pass[2];
          uint32_t ri[2];
#pragma unroll
          for (int u = 0; u < 2; u++) {
            pass[u] = p + u < end;
            ri[u] = 0;
            if (pass[u]) {
              const float4 e = __ldg(grid + p + u);
              const float dx = e.x - xs[0], dy = e.y - xs[1], dz = D == 3 ? e.z - xs[D - 1] : 0.0f;
              ri[u] = __float_as_uint(e.w);
              pass[u] = !(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > bd);
            }
          }
          p += 2;
#pragma unroll
          for (int u = 0; u < 2; u++) {
            const unsigned some = __ballot_sync(EJ_FULL_MASK, pass[u]);
            if (pass[u]) buf[held + __popc(some & ej_lanemask_lt())] = make_uint2((uint32_t)w + owner, ri[u]);
            held += __popc(some);
          }
          if (held > DJ_BUF - 64) {
            const uint32_t rows = dist_flush<D, COUNT_ONLY>(buf, held, R, S, rad.r2, out, cap, cursor);
            if (COUNT_ONLY) local += rows;
            held = 0;
          }
        }
      }
    }
  }
  if (held) {
    const uint32_t rows = dist_flush<D, COUNT_ONLY>(buf, held, R, S, rad.r2, out, cap, cursor);
    if (COUNT_ONLY) local += rows;
  }
  if (COUNT_ONLY) {
    unsigned long long total;
    ej_block_exclusive_sum<DJ_THREADS, unsigned long long>(local, warp_tmp, &total);
    if (threadIdx.x == 0 && total) atomicAdd(cursor, total);
  }
}

// ---- few S points ------------------------------------------------------------------
// Few S points are compared with every R point, which a lane brings in once: no grid.
// The grid of 2^24 R points costs 0.98 (2-D) and 1.55 ms (3-D; random atomics and
// stores), a compare with all of them 9.2 us per S point.
constexpr uint32_t DJ_FEW = 160;
template <int D>
constexpr uint32_t dist_few_most() { return D == 2 ? 112u : DJ_FEW; }

template <int D, bool COUNT_ONLY>
__global__ void __launch_bounds__(DJ_THREADS)
dist_few_kernel(const Point<D>* __restrict__ R, uint32_t nR, const Point<D>* __restrict__ S, uint32_t nS,
                DistRadius rad, typename RowOf<D>::type* __restrict__ out, uint64_t cap, unsigned long long* cursor) {
  __shared__ float4 points[DJ_FEW];  // coordinates and bound; a point that matches nothing has a negative bound
  __shared__ uint2 bufs[DJ_WARPS][DJ_BUF];
  __shared__ unsigned long long warp_tmp[DJ_WARPS + 1];
  const uint32_t lane = threadIdx.x & 31u;
  for (uint32_t i = threadIdx.x; i < nS; i += DJ_THREADS) {
    const Point<D> l = S[i];
    const bool ok = dist_finite<D>(l);
    double v[D];
#pragma unroll
    for (int d = 0; d < D; d++) v[d] = ok ? l.val[d] : 0.0;
    float x[D];
    const float bound = dist_screen_point<D>(v, rad.rho_up, x);
    points[i] = make_float4(x[0], x[1], D == 3 ? x[D - 1] : 0.0f, ok ? bound : -1.0f);
  }
  __syncthreads();
  uint2* buf = bufs[threadIdx.x >> 5];
  uint32_t held = 0;
  unsigned long long local = 0;
  constexpr int U = 2;  // R points per lane and step
  for (uint64_t w = (((uint64_t)blockIdx.x * DJ_THREADS + threadIdx.x) & ~31ull) * U; w < nR;
       w += (uint64_t)gridDim.x * DJ_THREADS * U) {
    float x[U][D];
    bool ok[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const uint64_t i = w + 32u * u + lane;
      ok[u] = i < nR;
#pragma unroll
      for (int d = 0; d < D; d++) x[u][d] = ok[u] ? __double2float_rn(__ldg(&R[i].val[d])) : 0.0f;
    }
    for (uint32_t s = 0; s < nS; s++) {
      const float4 l = points[s];
      bool pass[U], some = false;
#pragma unroll
      for (int u = 0; u < U; u++) {
        const float dx = x[u][0] - l.x, dy = x[u][1] - l.y, dz = D == 3 ? x[u][D - 1] - l.z : 0.0f;
        pass[u] = ok[u] && !(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > l.w);
        some |= pass[u];
      }
      if (!__any_sync(EJ_FULL_MASK, some)) continue;
#pragma unroll
      for (int u = 0; u < U; u++) {
        const unsigned b = __ballot_sync(EJ_FULL_MASK, pass[u]);
        if (pass[u]) buf[held + __popc(b & ej_lanemask_lt())] = make_uint2(s, (uint32_t)w + 32u * u + lane);
        held += __popc(b);
      }
      if (held > DJ_BUF - 64) {
        const uint32_t rows = dist_flush<D, COUNT_ONLY>(buf, held, R, S, rad.r2, out, cap, cursor);
        if (COUNT_ONLY) local += rows;
        held = 0;
      }
    }
  }
  if (held) {
    const uint32_t rows = dist_flush<D, COUNT_ONLY>(buf, held, R, S, rad.r2, out, cap, cursor);
    if (COUNT_ONLY) local += rows;
  }
  if (COUNT_ONLY) {
    unsigned long long total;
    ej_block_exclusive_sum<DJ_THREADS, unsigned long long>(local, warp_tmp, &total);
    if (threadIdx.x == 0 && total) atomicAdd(cursor, total);
  }
}

DistRadius dist_radius(double radius) {
  DistRadius r;
  r.rho = fabs(radius);
  const double w = 2.0 * r.rho;
  r.inv_w = w > 0.0 && w <= DBL_MAX ? 1.0 / w : 0.0;
  r.r2 = radius * radius;
  if (r.rho > (double)FLT_MAX) {
    r.rho_up = INFINITY;
  } else {
    r.rho_up = (float)r.rho;
    if ((double)r.rho_up < r.rho) r.rho_up = nextafterf(r.rho_up, INFINITY);
  }
  return r;
}

// buckets of a grid of n points: 2^bits, two to four per point
uint32_t dist_bits(uint64_t n) { return std::max(8u, ej_ceil_log2(n) + 1u); }

template <int D>
ej_status dist_few(ej_handle* h, const Point<D>* R, uint64_t nR, const Point<D>* S, uint32_t nS, const DistRadius& rad,
                   void* outv, uint64_t cap, bool count_only) {
  ej_phase_begin(h);
  for (int k = 1; k < EJ_PHASES; k++) ej_phase_mark(h, k);
  for (uint64_t r0 = 0; r0 < nR; r0 += DJ_FEW_RPIECE) {
    const uint32_t n = (uint32_t)std::min<uint64_t>(DJ_FEW_RPIECE, nR - r0);
    const unsigned blocks =
        (unsigned)std::min<uint64_t>(((uint64_t)n + 2 * DJ_THREADS - 1) / (2 * DJ_THREADS), (uint64_t)h->num_sms * 8);
    if (count_only)
      dist_few_kernel<D, true><<<blocks, DJ_THREADS, 0, h->stream>>>(R + r0, n, S, nS, rad, nullptr, 0, h->d_words);
    else
      dist_few_kernel<D, false><<<blocks, DJ_THREADS, 0, h->stream>>>(
          R + r0, n, S, nS, rad, static_cast<typename RowOf<D>::type*>(outv), cap, h->d_words);
    EJ_TRY(ej_check_launch(h, "dist_few_kernel"));
  }
  ej_phase_mark(h, EJ_PHASES);
  return EJ_OK;
}

template <int D>
ej_status dist_run(ej_handle* h, const void* Rv, uint64_t nR, const void* Sv, uint64_t nS, double radius, void* outv,
                   uint64_t cap, bool count_only, std::function<ej_status()>* crowded) {
  const Point<D>* R = static_cast<const Point<D>*>(Rv);
  const Point<D>* S = static_cast<const Point<D>*>(Sv);
  EJ_CUDA(h, cudaMemsetAsync(h->d_words, 0, (DJ_CROWD_WORD + 2) * sizeof(unsigned long long), h->stream));
  const DistRadius rad = dist_radius(radius);
  if (nR == 0 || nS == 0 || !(rad.r2 > 0.0)) return EJ_OK;
  if (nS <= dist_few_most<D>()) return dist_few<D>(h, R, nR, S, (uint32_t)nS, rad, outv, cap, count_only);
  // crowded buckets: few S points take all of the list's parts
  DistCrowd crowd;
  const uint64_t probes = std::min(nS, DJ_SPIECE);
  crowd.whole = (uint32_t)std::max(DJ_WHOLE, (probes + 31) / 32 * 8);
  crowd.parts = (uint32_t)std::max<uint64_t>(16, DJ_SPLIT / (probes << D));
  // R in pieces, smaller ones when memory is short
  uint64_t piece = std::min(nR, DJ_RPIECE);
  size_t ioff, coff, soff, scan_off, poff, goff;
  for (;; piece = (piece + 3) / 4) {
    const uint64_t nb = 1ull << dist_bits(piece);
    ej_plan_bytes p;
    ioff = p.add((DJ_SPLIT + crowd.whole) * sizeof(uint4));
    coff = p.add(nb * sizeof(uint32_t));
    soff = p.add((nb + 1) * sizeof(uint32_t));
    scan_off = p.add(ej_scan_scratch_bytes(nb));
    poff = p.add(piece * sizeof(uint2));
    goff = p.add(piece * sizeof(float4));
    const ej_status st = ej_arena_reserve(h, p.bytes);
    if (st == EJ_OK) break;
    if (st != EJ_ERR_NOMEM || piece <= DJ_LEAST_PIECE) return st;
  }
  h->last_error.clear();
  crowd.items = reinterpret_cast<uint4*>(ej_arena_at(h, ioff));
  crowd.header = reinterpret_cast<uint32_t*>(h->d_words + DJ_CROWD_WORD);
  uint32_t* count = reinterpret_cast<uint32_t*>(ej_arena_at(h, coff));
  uint32_t* start = reinterpret_cast<uint32_t*>(ej_arena_at(h, soff));
  uint2* place = reinterpret_cast<uint2*>(ej_arena_at(h, poff));
  float4* grid = reinterpret_cast<float4*>(ej_arena_at(h, goff));
  using Row = typename RowOf<D>::type;
  const unsigned cblocks = (unsigned)h->num_sms * 4;
  // the first piece's grid is the build phase; the probe (and any further pieces) the write phase
  ej_phase_begin(h);
  const bool pieces = nR > piece || nS > DJ_SPIECE;
  for (uint64_t r0 = 0; r0 < nR; r0 += piece) {
    const uint32_t n = (uint32_t)std::min<uint64_t>(piece, nR - r0);
    const uint32_t bits = dist_bits(n);
    const unsigned rblocks = (unsigned)std::min<uint64_t>(((uint64_t)n + 255) / 256, (uint64_t)h->num_sms * 8);
    EJ_CUDA(h, cudaMemsetAsync(count, 0, sizeof(uint32_t) << bits, h->stream));
    dist_cell_kernel<D><<<rblocks, 256, 0, h->stream>>>(R + r0, n, rad, bits, count, place);
    EJ_TRY(ej_check_launch(h, "dist_cell_kernel"));
    EJ_TRY(ej_scan_u32_u32(h, count, 1ull << bits, start, ej_arena_at(h, scan_off)));
    dist_place_kernel<D><<<rblocks, 256, 0, h->stream>>>(R + r0, n, place, start, grid);
    EJ_TRY(ej_check_launch(h, "dist_place_kernel"));
    if (r0 == 0)
      for (int k = 1; k < EJ_PHASES; k++) ej_phase_mark(h, k);
    for (uint64_t s0 = 0; s0 < nS; s0 += DJ_SPIECE) {
      const uint32_t ns = (uint32_t)std::min<uint64_t>(DJ_SPIECE, nS - s0);
      if (pieces) EJ_CUDA(h, cudaMemsetAsync(crowd.header, 0, 2 * sizeof(unsigned long long), h->stream));
      const unsigned sblocks =
          (unsigned)std::min<uint64_t>(((uint64_t)ns + DJ_THREADS - 1) / DJ_THREADS, (uint64_t)h->num_sms * 8);
      if (count_only)
        dist_probe_kernel<D, true><<<sblocks, DJ_THREADS, 0, h->stream>>>(R + r0, S + s0, ns, start, grid, bits, rad,
                                                                          crowd, nullptr, 0, h->d_words);
      else
        dist_probe_kernel<D, false><<<sblocks, DJ_THREADS, 0, h->stream>>>(
            R + r0, S + s0, ns, start, grid, bits, rad, crowd, static_cast<Row*>(outv), cap, h->d_words);
      EJ_TRY(ej_check_launch(h, "dist_probe_kernel"));
      const auto rest = [=]() -> ej_status {
        if (count_only)
          dist_crowd_kernel<D, true><<<cblocks, DJ_THREADS, 0, h->stream>>>(R + r0, S + s0, grid, crowd, rad, nullptr,
                                                                            0, h->d_words);
        else
          dist_crowd_kernel<D, false><<<cblocks, DJ_THREADS, 0, h->stream>>>(
              R + r0, S + s0, grid, crowd, rad, static_cast<Row*>(outv), cap, h->d_words);
        return ej_check_launch(h, "dist_crowd_kernel");
      };
      // one piece: the caller launches it if its read-back finds items (a launch that
      // finds none costs 5 us, of a call of 110); phase timing wants it in place
      if (pieces || h->timing)
        EJ_TRY(rest());
      else
        *crowded = rest;
    }
  }
  ej_phase_mark(h, EJ_PHASES);
  return EJ_OK;
}

ej_status dist_entry(ej_handle* h, uint32_t dims, const void* R, uint64_t nR, const void* S, uint64_t nS,
                     double radius, void* out, uint64_t cap, uint64_t* out_count, bool count_only) {
  EJ_TRY(ej_begin(h));
  if (dims != 2 && dims != 3) return ej_fail(h, EJ_ERR_INVALID, "dims must be 2 or 3 (got %u)", dims);
  if (!out_count) return ej_fail(h, EJ_ERR_INVALID, "out_count is NULL");
  if ((nR && !R) || (nS && !S)) return ej_fail(h, EJ_ERR_INVALID, "point array is NULL");
  if (!count_only && cap && !out)
    return ej_fail(h, EJ_ERR_INVALID, "out is NULL with capacity %llu", (unsigned long long)cap);
  if (((uintptr_t)R | (uintptr_t)S | (uintptr_t)out) % 8)
    return ej_fail(h, EJ_ERR_INVALID, "point and row arrays must be 8-byte aligned");
  std::function<ej_status()> crowded;
  EJ_TRY(dims == 2 ? dist_run<2>(h, R, nR, S, nS, radius, out, cap, count_only, &crowded)
                   : dist_run<3>(h, R, nR, S, nS, radius, out, cap, count_only, &crowded));
  uint64_t count = 0;
  EJ_TRY(ej_finish(h, &count));
  if (crowded && h->h_words[DJ_CROWD_WORD] != 0) {
    EJ_TRY(crowded());
    EJ_TRY(ej_finish(h, &count));
  }
  *out_count = count;
  return count_only ? EJ_OK : ej_capacity_result(h, count, cap);
}

}  // namespace

extern "C" ej_status ej_distance_join(ej_handle* h, uint32_t dims, const void* R, uint64_t nR, const void* S,
                                      uint64_t nS, double radius, void* out, uint64_t out_cap, uint64_t* out_count) {
  return dist_entry(h, dims, R, nR, S, nS, radius, out, out_cap, out_count, false);
}

extern "C" ej_status ej_distance_join_count(ej_handle* h, uint32_t dims, const void* R, uint64_t nR, const void* S,
                                            uint64_t nS, double radius, uint64_t* out_count) {
  return dist_entry(h, dims, R, nR, S, nS, radius, nullptr, 0, out_count, true);
}
