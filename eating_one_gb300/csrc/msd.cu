// msd.cu - the hash-sorted table build of large hash tables: two unordered
// most-significant-digit radix passes, then one shared-memory sort per bucket.
//
// The table (hash_join.cu) needs R ordered by hash32(val), with equal keys
// adjacent; the order among rows of one key is never used.  So no pass has to
// be stable, and the sort can go most-significant digit first:
//   1. an unordered radix pass by hash bits 24..31 (256 segments);
//   2. an unordered segmented pass by bits 16..23 inside every segment (65536
//      buckets of about |R|/65536 rows) - its tile descriptors are laid out on
//      the device from the first pass's offsets, so the host never waits;
//   3. one CTA per group of consecutive buckets (about 2048 rows) orders the
//      group by its remaining hash bits in shared memory (a counting pass by
//      12 of them into sub-buckets of a few rows, then every row ranked within
//      its sub-bucket) and writes each row once, to its place in the table's
//      two columns rkey[]/rval[].
// Three passes over R instead of the four of an LSD sort, none with the
// ballot ranking a stable pass needs.  A bucket too large for shared memory
// (many rows of few keys) is sorted by its CTA through global memory
// instead, one 8-bit digit at a time.
//
// The slot tables of large build sides (slot_table.cuh) share the two passes:
// their third step builds each bucket group's part of the slot array in shared
// memory and writes it out whole (msd_slots_kernel).
//
// Replaces, for the hash join's build side, the reference's partitioning of
// R (joins/hashJoin_gpu/main_street/partitioning.cu:133-271, rcount_partitioning
// + rpartitioning, one 6-bit digit per pass with a host round trip each).
#include <algorithm>

#include "ej_device.cuh"
#include "msd.cuh"
#include "slot_table.cuh"

namespace {

constexpr uint32_t MSD_BUCKET_BITS = 16;
constexpr uint32_t MSD_BUCKETS = 1u << MSD_BUCKET_BITS;
constexpr int LS_THREADS = 256;
constexpr int LS_CAP = 3072;                 // rows of a bucket group sorted in shared memory
constexpr int LS_PER = LS_CAP / LS_THREADS;  // rows per thread
constexpr uint32_t LS_ROWS = 2048;           // bucket groups aim at this many rows
constexpr uint32_t LS_DIGIT_BITS = 12;       // digit of the counting pass in shared memory
constexpr uint32_t LS_DIGITS = 1u << LS_DIGIT_BITS;
constexpr uint32_t LS_MAX_GROUP_BITS = 4;    // groups of at most 16 buckets
constexpr uint32_t LS_SMALL = 32;            // sub-buckets up to this size: each row ranked on its own

// the first pass's digit d (cells d * ntiles1 + t) is segment d: its start,
// its tiles, and the first tile of the second pass it gets
struct MsdSegments {
  uint32_t start[257];  // start[256] = n
  uint32_t end[256];    // start[d] + rows of segment d
  uint32_t tbase[257];  // first tile of the second pass; tbase[256] = tiles in use
};

__global__ void __launch_bounds__(256) msd_segments_kernel(const uint32_t* __restrict__ offs1, uint32_t ntiles1,
                                                           uint64_t n, MsdSegments* __restrict__ seg) {
  __shared__ uint32_t tmp[256 / 32 + 1], first[256];
  const uint32_t d = threadIdx.x;
  // clamped and made monotone, so that offsets left too small by a timed-out scan
  // still give ordered segments inside [0, n), of no more tiles than planned
  first[d] = min(offs1[(uint64_t)d * ntiles1], (uint32_t)n);
  for (uint32_t step = 1; step < 256; step <<= 1) {
    __syncthreads();
    const uint32_t before = d >= step ? first[d - step] : 0u;
    __syncthreads();
    first[d] = max(first[d], before);
  }
  __syncthreads();
  const uint32_t s = first[d];
  const uint32_t e = d < 255 ? first[d + 1] : (uint32_t)n;
  const uint32_t tiles = (e - s + EJ_RX_TILE - 1) / EJ_RX_TILE;
  uint32_t total;
  const uint32_t base = ej_block_exclusive_sum<256, uint32_t>(tiles, tmp, &total);
  seg->start[d] = s;
  seg->tbase[d] = base;
  seg->end[d] = e;
  if (d == 255) {
    seg->start[256] = (uint32_t)n;
    seg->tbase[256] = total;
  }
}

// descriptor of every tile of the second pass: tile t of segment d covers
// rows start[d] + 4096 t ... and owns cells 256 tbase[d] + t + k tiles_d
// (digit k); tiles past those in use are empty and own cells past them all
__global__ void __launch_bounds__(256) msd_tiles_kernel(const MsdSegments* __restrict__ seg,
                                                        ej_rx_tile* __restrict__ desc, uint32_t max_tiles) {
  __shared__ uint32_t tb[257];
  for (uint32_t i = threadIdx.x; i < 257; i += blockDim.x) tb[i] = seg->tbase[i];
  __syncthreads();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= max_tiles) return;
  const uint32_t used = tb[256];
  ej_rx_tile t;
  t.pad = 0;
  if (i < used) {
    uint32_t lo = 0, hi = 256;  // the segment d with tb[d] <= i < tb[d + 1]
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (tb[mid] <= i) lo = mid; else hi = mid;
    }
    const uint32_t d = lo, k = i - tb[d], tiles = tb[d + 1] - tb[d];
    const uint32_t s = seg->start[d] + k * EJ_RX_TILE, e = seg->end[d];
    t.start = s;
    t.n = min((uint32_t)EJ_RX_TILE, e - s);
    t.cell0 = 256u * tb[d] + k;
    t.stride = tiles;
  } else {
    t.start = 0;
    t.n = 0;
    t.cell0 = 256u * i;  // i >= used: past every cell of the tiles in use
    t.stride = 1;
  }
  desc[i] = t;
}

// bucket (d1, d2) starts where the second pass put digit d2 of segment d1's
// first tile; bstart[65536] = n
__global__ void __launch_bounds__(256) msd_bucket_kernel(const MsdSegments* __restrict__ seg,
                                                         const uint32_t* __restrict__ offs2, uint64_t n,
                                                         uint32_t* __restrict__ bstart) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b > MSD_BUCKETS) return;
  if (b == MSD_BUCKETS) {
    bstart[b] = (uint32_t)n;
    return;
  }
  const uint32_t d1 = b >> 8, d2 = b & 255u;
  const uint32_t tiles = seg->tbase[d1 + 1] - seg->tbase[d1];
  bstart[b] = tiles ? offs2[256ull * seg->tbase[d1] + (uint64_t)d2 * tiles] : seg->start[d1];
}

struct LsSmem {
  uint2 row[LS_CAP];              // the group's tuples in digit order
  uint32_t hsh[LS_CAP];           // their hashes
  uint32_t cnt[LS_DIGITS + 1];    // digit counts, then digit starts (cnt[LS_DIGITS] = rows)
  uint32_t cnt2[256];             // counts of a long sub-bucket's remaining bits (at most 8 of them)
  uint32_t big[LS_CAP / (LS_SMALL + 1) + 1];  // digits whose sub-bucket is longer than LS_SMALL
  uint32_t warp_tmp[LS_THREADS / 32 + 1];
  uint32_t nbig;
};

// Digit d's counter sits at ls_at(d) = d ^ ((d >> 5) & 31), a permutation
// within each 32-counter row: the scan below, where thread t takes digits
// 16t .. 16t + 15, and the placement, where a warp's lanes take consecutive
// rows of non-decreasing digits, both read 32 distinct banks per instruction
// (a plain layout gave the scan 16-way conflicts).  Index LS_DIGITS (the
// total) maps to itself.
__device__ __forceinline__ uint32_t ls_at(uint32_t d) { return d ^ ((d >> 5) & 31u); }

// exclusive sum in place of the LS_DIGITS counters (at ls_at(d)); c at
// LS_DIGITS = total.  Every thread, LS_DIGITS / LS_THREADS consecutive
// digits; the counters are read twice rather than held, as the caller's rows
// occupy the registers
__device__ __forceinline__ void ls_scan_digits(uint32_t* c, uint32_t* warp_tmp) {
  constexpr int PER = LS_DIGITS / LS_THREADS;
  const uint32_t d0 = threadIdx.x * PER;
  uint32_t sum = 0;
#pragma unroll
  for (int i = 0; i < PER; i++) sum += c[ls_at(d0 + i)];
  uint32_t total;
  uint32_t run = ej_block_exclusive_sum<LS_THREADS, uint32_t>(sum, warp_tmp, &total);
#pragma unroll
  for (int i = 0; i < PER; i++) {
    const uint32_t x = c[ls_at(d0 + i)];
    c[ls_at(d0 + i)] = run;
    run += x;
  }
  if (threadIdx.x == 0) c[LS_DIGITS] = total;
  __syncthreads();
}

// The CTA sorts the rows [a, a + len) of `src` by hash bits 0..7 (all of them
// share bits 8..31) into rkey/rval at the same positions: a counting sort
// through global memory (order among equal hashes, which are equal keys,
// unspecified).  Shared counters: sm.cnt2.  `src` was written earlier in this
// launch (by this CTA), so it is read through L2 (__ldcg), never through the
// read-only cache, which another CTA on the SM may have filled with the same
// lines before they were written; a stale line would make the two loops
// below see different rows.
__device__ void ls_digit_global(LsSmem& sm, const ej_tuple* src, uint64_t a, uint32_t len,
                                int32_t* __restrict__ rkey, int32_t* __restrict__ rval) {
  sm.cnt2[threadIdx.x] = 0;
  __syncthreads();
  const uint2* s2 = reinterpret_cast<const uint2*>(src);
  for (uint32_t j = threadIdx.x; j < len; j += LS_THREADS)
    atomicAdd(&sm.cnt2[ej_hash32(__ldcg(s2 + a + j).y) & 255u], 1u);
  __syncthreads();
  uint32_t c = sm.cnt2[threadIdx.x];
  uint32_t total;
  const uint32_t ex = ej_block_exclusive_sum<LS_THREADS, uint32_t>(c, sm.warp_tmp, &total);
  sm.cnt2[threadIdx.x] = ex;
  __syncthreads();
  for (uint32_t j = threadIdx.x; j < len; j += LS_THREADS) {
    const uint2 x = __ldcg(s2 + a + j);
    const uint32_t p = atomicAdd(&sm.cnt2[ej_hash32(x.y) & 255u], 1u);
    if (p < len) {  // always; a guard that keeps every store inside the range
      rkey[a + p] = (int32_t)x.x;
      rval[a + p] = (int32_t)x.y;
    }
  }
  __syncthreads();
}

// A bucket larger than shared memory: by bits 8..15 from `in` into `tmp`
// (same positions), then every sub-bucket by bits 0..7 into the columns.
// Shared counters: sm.cnt (256 of them, with their starts in cnt[256 ...]).
__device__ void ls_bucket_global(LsSmem& sm, const ej_tuple* __restrict__ in, ej_tuple* __restrict__ tmp,
                                 uint64_t lo, uint32_t m, int32_t* __restrict__ rkey, int32_t* __restrict__ rval) {
  const uint2* s2 = reinterpret_cast<const uint2*>(in);
  uint2* t2 = reinterpret_cast<uint2*>(tmp);
  uint32_t* cur = sm.cnt;
  uint32_t* st = sm.cnt + 256;  // 257 starts
  cur[threadIdx.x] = 0;
  __syncthreads();
  for (uint32_t j = threadIdx.x; j < m; j += LS_THREADS) atomicAdd(&cur[(ej_hash32(s2[lo + j].y) >> 8) & 255u], 1u);
  __syncthreads();
  {
    const uint32_t c = cur[threadIdx.x];
    uint32_t total;
    const uint32_t ex = ej_block_exclusive_sum<LS_THREADS, uint32_t>(c, sm.warp_tmp, &total);
    st[threadIdx.x] = ex;
    cur[threadIdx.x] = ex;
    if (threadIdx.x == 0) st[256] = total;
    __syncthreads();
  }
  for (uint32_t j = threadIdx.x; j < m; j += LS_THREADS) {
    const uint2 x = s2[lo + j];
    const uint32_t p = atomicAdd(&cur[(ej_hash32(x.y) >> 8) & 255u], 1u);
    if (p < m) t2[lo + p] = x;  // always; a guard that keeps every store inside the range
  }
  __syncthreads();  // the CTA's own global writes are visible to it past the barrier
  for (uint32_t s = 0; s < 256; s++) {
    const uint32_t a = st[s], len = st[s + 1] - a;
    if (len) ls_digit_global(sm, tmp, lo + a, len, rkey, rval);
  }
}

// The CTA sorts the m <= LS_CAP rows [lo, lo + m) of `in`, which share hash
// bits low_bits..31 (LS_DIGIT_BITS <= low_bits <= LS_DIGIT_BITS + 8), into the
// columns by the full hash: a counting pass by the LS_DIGIT_BITS bits below
// low_bits groups the rows into sub-buckets of a few rows each; every row's
// place in its sub-bucket is the number of rows there with a smaller hash
// (or the same hash and an earlier slot), so each row is written once, at
// its final position.  Long sub-buckets (many rows of few keys) are sorted
// by the whole CTA instead: a counting sort by their remaining bits.
//
// PER: row slots per thread (m <= PER * LS_THREADS), so that a small group
// does not pay for the slots of the largest; up to 9 slots the rows' hashes
// stay in registers between the ranking and the placement (beyond that they
// are computed again, for want of registers).
template <int PER>
__device__ void ls_sort_smem(LsSmem& sm, const ej_tuple* __restrict__ in, uint64_t lo, uint32_t m,
                             uint32_t low_bits, int32_t* __restrict__ rkey, int32_t* __restrict__ rval) {
  constexpr bool KEEP = PER <= 9;
  const unsigned t = threadIdx.x;
  const uint32_t sh = low_bits - LS_DIGIT_BITS;  // bits under the digit
  for (uint32_t i = t; i < LS_DIGITS / 4; i += LS_THREADS) reinterpret_cast<uint4*>(sm.cnt)[i] = make_uint4(0, 0, 0, 0);
  if (t == 0) sm.nbig = 0;
  __syncthreads();
  // 1. rows into registers (coalesced), ranked within their digit
  const uint2* src = reinterpret_cast<const uint2*>(in) + lo;
  uint2 v[PER];
  uint32_t rk[PER], hk[KEEP ? PER : 1];
#pragma unroll
  for (int i = 0; i < PER; i++) {
    const uint32_t j = t + (uint32_t)i * LS_THREADS;
    if (j < m) v[i] = __ldcs(src + j);
  }
#pragma unroll
  for (int i = 0; i < PER; i++)
    if (t + (uint32_t)i * LS_THREADS < m) {
      const uint32_t hv = ej_hash32(v[i].y);
      if (KEEP) hk[KEEP ? i : 0] = hv;
      rk[i] = atomicAdd(&sm.cnt[ls_at((hv >> sh) & (LS_DIGITS - 1))], 1u);
    }
  __syncthreads();
  ls_scan_digits(sm.cnt, sm.warp_tmp);
  // 2. every row to its digit's sub-bucket
#pragma unroll
  for (int i = 0; i < PER; i++)
    if (t + (uint32_t)i * LS_THREADS < m) {
      const uint32_t hv = KEEP ? hk[KEEP ? i : 0] : ej_hash32(v[i].y);
      const uint32_t p = sm.cnt[ls_at((hv >> sh) & (LS_DIGITS - 1))] + rk[i];
      sm.row[p] = v[i];
      sm.hsh[p] = hv;
    }
  __syncthreads();
  // 3. each row of a short sub-bucket straight to its place (the lanes of a
  //    warp take consecutive slots, so their stores stay within a few rows
  //    of each other); long sub-buckets are listed for step 4
  for (uint32_t p = t; p < m; p += LS_THREADS) {
    const uint32_t hv = sm.hsh[p];
    const uint32_t d = (hv >> sh) & (LS_DIGITS - 1);
    const uint32_t a = sm.cnt[ls_at(d)], e = sm.cnt[ls_at(d + 1)];
    if (e - a > LS_SMALL) {
      if (p == a) sm.big[atomicAdd(&sm.nbig, 1u)] = d;
      continue;
    }
    uint32_t r = a;
    for (uint32_t q = a; q < e; q++) {
      const uint32_t x = sm.hsh[q];
      r += (x < hv || (x == hv && q < p)) ? 1u : 0u;
    }
    const uint2 row = sm.row[p];
    rkey[lo + r] = (int32_t)row.x;
    rval[lo + r] = (int32_t)row.y;
  }
  __syncthreads();
  // 4. long sub-buckets: a counting sort by the bits under the digit,
  //    straight to the columns
  const uint32_t nbig = sm.nbig, rmask = (1u << sh) - 1u;
  for (uint32_t q = 0; q < nbig; q++) {
    const uint32_t d = sm.big[q];
    const uint32_t a = sm.cnt[ls_at(d)], len = sm.cnt[ls_at(d + 1)] - a;
    sm.cnt2[t] = 0;
    __syncthreads();
    for (uint32_t j = t; j < len; j += LS_THREADS) atomicAdd(&sm.cnt2[sm.hsh[a + j] & rmask], 1u);
    __syncthreads();
    const uint32_t c = sm.cnt2[t];
    uint32_t total;
    const uint32_t ex = ej_block_exclusive_sum<LS_THREADS, uint32_t>(c, sm.warp_tmp, &total);
    sm.cnt2[t] = ex;
    __syncthreads();
    for (uint32_t j = t; j < len; j += LS_THREADS) {
      const uint2 x = sm.row[a + j];
      const uint32_t p = a + atomicAdd(&sm.cnt2[sm.hsh[a + j] & rmask], 1u);
      rkey[lo + p] = (int32_t)x.x;
      rval[lo + p] = (int32_t)x.y;
    }
    __syncthreads();
  }
  __syncthreads();  // shared memory is reused by the caller's next range
}

// ls_sort_smem with the fewest row slots per thread that hold m rows (groups
// aim at LS_ROWS = 8 slots' worth; 9 takes most of those a little over)
__device__ __forceinline__ void ls_sort_rows(LsSmem& sm, const ej_tuple* __restrict__ in, uint64_t lo, uint32_t m,
                                             uint32_t low_bits, int32_t* __restrict__ rkey,
                                             int32_t* __restrict__ rval) {
  if (m <= 4u * LS_THREADS)
    ls_sort_smem<4>(sm, in, lo, m, low_bits, rkey, rval);
  else if (m <= 8u * LS_THREADS)
    ls_sort_smem<8>(sm, in, lo, m, low_bits, rkey, rval);
  else if (m <= 9u * LS_THREADS)
    ls_sort_smem<9>(sm, in, lo, m, low_bits, rkey, rval);
  else
    ls_sort_smem<LS_PER>(sm, in, lo, m, low_bits, rkey, rval);
}

// One CTA per group of 2^g consecutive buckets (b = top 16 hash bits), whose
// rows [bstart[b0], bstart[b0 + 2^g]) of `in` share hash bits 16 + g .. 31:
// into the columns ordered by the full hash.  A group larger than shared
// memory goes bucket by bucket, and a bucket larger than shared memory
// through global memory.
__global__ void __launch_bounds__(LS_THREADS, 4)
msd_local_kernel(const ej_tuple* __restrict__ in, ej_tuple* __restrict__ tmp, const uint32_t* __restrict__ bstart,
                 uint32_t g, int32_t* __restrict__ rkey, int32_t* __restrict__ rval) {
  extern __shared__ __align__(16) unsigned char ls_smem_raw[];
  LsSmem& sm = *reinterpret_cast<LsSmem*>(ls_smem_raw);
  // bounds clamped to [0, n) and ordered (they are, unless a scan timed out)
  const uint32_t n = bstart[MSD_BUCKETS];
  const uint32_t b0 = blockIdx.x << g, b1 = b0 + (1u << g);
  const uint32_t lo = min(bstart[b0], n);
  const uint32_t hi = max(min(bstart[b1], n), lo);
  if (hi - lo <= (uint32_t)LS_CAP) {
    if (hi > lo) ls_sort_rows(sm, in, lo, hi - lo, MSD_BUCKET_BITS + g, rkey, rval);
    return;
  }
  for (uint32_t b = b0; b < b1; b++) {
    const uint32_t blo = max(min(bstart[b], n), lo);
    const uint32_t bhi = min(max(min(bstart[b + 1], n), blo), hi);
    if (bhi - blo > (uint32_t)LS_CAP)
      ls_bucket_global(sm, in, tmp, blo, bhi - blo, rkey, rval);
    else if (bhi > blo)
      ls_sort_rows(sm, in, blo, bhi - blo, MSD_BUCKET_BITS, rkey, rval);
  }
}

// ---- slot tables of large build sides -----------------------------------------------
// A group of 2^g buckets holds a contiguous range of hashes, so with as many
// pairs per group (pp) everywhere, the group's keys have their homes in its own
// pp pairs.  One CTA claims the group's slots in shared memory, gives the keys
// with several rows their runs (words [lo + lo / 31 + 4 group, ...) of rkey[], where
// the group's rows begin at lo: room for its rows and the long runs' counts), and
// writes slots and runs out.  A key whose walk passes the group's end is
// spilled: its rows go to a list that the passes below insert into the finished
// array (a row or two per group at half load; its run comes from the group's
// own words).  Random slot updates through L2 (slot_insert_kernel) run at 40 to
// 60 G rows/s; here they stay in shared memory and the slots leave in
// coalesced stores.  Bound by the shared memory's compare-and-swaps (random
// 8-byte words, a warp's longest walk of some rounds): 2^24 rows in 178 us, where
// the local sort and the directory or bucket launches took 230 to 250 (200 with
// walks that all begin with a pair's first slot; four CTAs an SM with the runs'
// cursors in shared memory too were level with six).  The build of a 2^24-row
// table in all: 420 us (432 with the sort), and the probes of unique keys then take
// 665 us instead of 1052.
constexpr uint32_t SB_PER = 12;           // rows per thread kept in registers (groups up to 3072 rows)
constexpr uint32_t SB_BIG = 8;            // rows per thread and step of larger groups
constexpr uint32_t SB_SPILLED = 0xFFFFu;  // a row's slot within its group (of 4098 at most): walked past the end
constexpr uint32_t SB_NONE = 0xFFFEu;     // no row
constexpr int SB_BLOCKS = 6;  // CTAs per SM

// `rows` rows of hash hv into the group's array (pairs p0 ..., `end` slots): their
// slot, and the first one's rank among their key's rows.  No slot for a row of another group: there is
// none unless a scan of the passes gave up waiting and left wrong bounds, which
// may then overlap; taking only its own rows, each once, a group stays within
// its run words, and the spilled rows within their list.
__device__ __forceinline__ uint32_t sb_claim(unsigned long long* slot, uint32_t hv, uint32_t npairs, uint32_t p0,
                                             uint32_t end, uint32_t* rank, uint32_t rows = 1u) {
  const uint32_t y = hv << 1 | 1u;
  *rank = 0u;
  const uint32_t home = 2u * (ej_home_pair(hv, npairs) - p0);
  if (home >= end) return SB_NONE;
  for (uint32_t s = home + (hv & 1u); s < end; s = ej_next_slot(s, hv, 0xFFFFFFFFu)) {
    const unsigned long long old = atomicCAS(slot + s, 0ull, (unsigned long long)y << 32 | rows);
    if (old == 0ull) return s;
    if ((uint32_t)(old >> 32) == y) {
      *rank = atomicAdd(reinterpret_cast<uint32_t*>(slot + s), rows);
      return s;
    }
  }
  return SB_SPILLED;
}

// that slot again, once the slots have their final form
__device__ __forceinline__ uint32_t sb_find(const unsigned long long* slot, uint32_t hv, uint32_t npairs, uint32_t p0,
                                            uint32_t end) {
  for (uint32_t s = 2u * (ej_home_pair(hv, npairs) - p0); s < end; s++)
    if (((uint32_t)(slot[s] >> 32) | 1u) == (hv << 1 | 1u) && slot[s] != 0ull) return s;
  return SB_SPILLED;
}

// a row to its place once the runs are laid out: its key into the slot, or to
// its place in the run
__device__ __forceinline__ void sb_place(unsigned long long* slot, uint32_t s, uint32_t rank, int32_t key,
                                         int32_t* __restrict__ rkey) {
  const unsigned long long w = slot[s];
  if (w >> 32 & 1u)
    rkey[((uint32_t)w >> 5) + rank] = key;
  else
    reinterpret_cast<int32_t*>(slot + s)[0] = key;
}

__global__ void __launch_bounds__(LS_THREADS, SB_BLOCKS)
msd_slots_kernel(const ej_tuple* __restrict__ in, const uint32_t* __restrict__ bstart, uint32_t g, uint32_t npairs,
                 uint32_t pp, uint4* __restrict__ pair, int32_t* __restrict__ rkey, uint32_t* __restrict__ gcursor,
                 uint2* __restrict__ spill, uint32_t* __restrict__ nspill, uint32_t* __restrict__ ranks,
                 const uint32_t* __restrict__ gave_up) {
  extern __shared__ __align__(16) unsigned char sb_smem_raw[];
  unsigned long long* slot = reinterpret_cast<unsigned long long*>(sb_smem_raw);
  __shared__ uint32_t s_runs;
  const uint32_t t = threadIdx.x, lane = t & 31u, end = 2u * pp, p0 = blockIdx.x * pp;
  // bounds clamped to [0, n) and ordered (they are, unless a scan timed out)
  const uint32_t n = bstart[MSD_BUCKETS];
  const uint32_t lo = min(bstart[blockIdx.x << g], n);
  uint32_t m = max(min(bstart[(blockIdx.x + 1u) << g], n), lo) - lo;
  // a scan of this build's passes gave up waiting: the call reports it, and the
  // bounds and rows are not to be relied on, so the table stays empty.  (Not the
  // handle's status: it holds an earlier asynchronous call's code until it is read.)
  if (*gave_up) m = 0u;
  // the group's words begin at a multiple of four, so that runs of four rows
  // throughout (one 16-byte load each) stay aligned
  const uint32_t words0 = ((lo + lo / 31u) & ~3u) + 4u * blockIdx.x;
  const int2* rows = reinterpret_cast<const int2*>(in) + lo;
  for (uint32_t i = t; i < pp; i += LS_THREADS) reinterpret_cast<uint4*>(slot)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (t == 0) s_runs = 0u;
  __syncthreads();
  // 1. every row's slot, claimed or counted in; rows past the group's end listed
  int32_t key[SB_PER];
  uint32_t at[SB_PER];  // slot | rank << 16
#pragma unroll
  for (uint32_t q = 0; q < SB_PER; q++) {  // (a group may have no rows)
    key[q] = 0;
    at[q] = SB_NONE;
  }
  const bool big = m > SB_PER * LS_THREADS;
  // more rows than the registers hold: many of few keys, so the rows of a key in a
  // warp go together, eight steps' loads at a time (a count of 3 M rows of one key
  // 12.4 ms when each row claims for itself, 5.8 here, 11.0 with the sorted table;
  // 2^24 rows of 50 keys 2.76, 1.22 and 2.91)
  for (uint32_t j0 = 0; big && j0 < m; j0 += SB_BIG * LS_THREADS) {
    int2 r[SB_BIG];
#pragma unroll
    for (uint32_t q = 0; q < SB_BIG; q++) {
      const uint32_t j = j0 + t + q * LS_THREADS;
      r[q] = j < m ? __ldcs(rows + j) : make_int2(0, 0);
    }
#pragma unroll
    for (uint32_t q = 0; q < SB_BIG; q++) {
      const uint32_t j = j0 + t + q * LS_THREADS;
      const uint32_t hv = ej_hash32((uint32_t)r[q].y);
      const unsigned peers = __match_any_sync(EJ_FULL_MASK, hv) & __ballot_sync(EJ_FULL_MASK, j < m);
      const int leader = peers ? __ffs(peers) - 1 : 0;
      uint32_t s = SB_NONE, rank = 0;
      if (j < m && (int)lane == leader) s = sb_claim(slot, hv, npairs, p0, end, &rank, __popc(peers));
      s = __shfl_sync(EJ_FULL_MASK, s, leader);
      rank = __shfl_sync(EJ_FULL_MASK, rank, leader) + __popc(peers & ej_lanemask_lt());
      if (j >= m) continue;
      if (s == SB_SPILLED) spill[atomicAdd(nspill, 1u)] = make_uint2((uint32_t)r[q].x, (uint32_t)r[q].y);
      ranks[lo + j] = rank;
    }
  }
  if (!big) {
#pragma unroll
    for (uint32_t q = 0; q < SB_PER; q++) {  // the loads together
      const uint32_t j = t + q * LS_THREADS;
      const int2 r = j < m ? __ldcs(rows + j) : make_int2(0, 0);
      key[q] = r.x;
      at[q] = (uint32_t)r.y;
    }
    // one row after the other, each warp until its longest walk ends (all rows'
    // walks advancing together took 2.5 times the instructions: 464 us at 2^24)
#pragma unroll
    for (uint32_t q = 0; q < SB_PER; q++) {
      const uint32_t j = t + q * LS_THREADS, val = at[q];
      at[q] = SB_NONE;
      if (j >= m) continue;
      uint32_t rank;
      const uint32_t s = sb_claim(slot, ej_hash32(val), npairs, p0, end, &rank);
      if (s == SB_SPILLED) spill[atomicAdd(nspill, 1u)] = make_uint2((uint32_t)key[q], val);
      at[q] = s | rank << 16;
    }
  }
  __syncthreads();
  // 2. the final form of every slot but the single rows' keys; runs laid out
  for (uint32_t s0 = 0; s0 < end; s0 += LS_THREADS) {
    const uint32_t s = s0 + t;
    const unsigned long long w = s < end ? slot[s] : 0ull;
    const uint32_t c = (uint32_t)w, y = (uint32_t)(w >> 32);
    const bool run = y != 0u && (c > 1u || y == 1u);
    const uint32_t need = run ? c + (c >= 31u ? 1u : 0u) : 0u;
    if (y != 0u && !run) slot[s] = (unsigned long long)(y & ~1u) << 32;
    if (!__any_sync(EJ_FULL_MASK, run)) continue;
    const uint32_t incl = ej_warp_inclusive_sum(need);
    uint32_t first = 0;
    if (lane == 31u) first = atomicAdd(&s_runs, incl);
    first = words0 + __shfl_sync(EJ_FULL_MASK, first, 31) + incl - need;
    if (!run) continue;
    if (c >= 31u) rkey[first++] = (int32_t)c;
    slot[s] = (unsigned long long)y << 32 | (first << 5 | min(c, 31u));
  }
  __syncthreads();
  // 3. every row to its slot or run
  if (!big) {
#pragma unroll
    for (uint32_t q = 0; q < SB_PER; q++)
      if ((at[q] & 0xFFFFu) < SB_NONE) sb_place(slot, at[q] & 0xFFFFu, at[q] >> 16, key[q], rkey);
  } else {
    for (uint32_t j0 = t; j0 < m; j0 += SB_BIG * LS_THREADS) {
      int2 r[SB_BIG];
      uint32_t rank[SB_BIG];
#pragma unroll
      for (uint32_t q = 0; q < SB_BIG; q++) {
        const uint32_t j = j0 + q * LS_THREADS;
        r[q] = j < m ? __ldg(rows + j) : make_int2(0, 0);
        rank[q] = j < m ? ranks[lo + j] : 0u;
      }
#pragma unroll
      for (uint32_t q = 0; q < SB_BIG; q++) {
        if (j0 + q * LS_THREADS >= m) continue;
        const uint32_t s = sb_find(slot, ej_hash32((uint32_t)r[q].y), npairs, p0, end);
        if (s != SB_SPILLED) sb_place(slot, s, rank[q], r[q].x, rkey);
      }
    }
  }
  __syncthreads();
  for (uint32_t i = t; i < pp; i += LS_THREADS) pair[p0 + i] = reinterpret_cast<const uint4*>(slot)[i];
  if (t == 0) gcursor[blockIdx.x] = words0 + s_runs;
}

// The spilled rows, by slot_table.cuh's steps on the whole array; their runs come
// from their home groups' words.  A spilled row's key is in none of its group's
// slots from its home on, so its walk starts behind the group, and passes the
// slots that hold other keys for good eight at a time (one compare-and-swap a
// slot from the home on took 19 us for a few hundred rows).
__global__ void __launch_bounds__(256)
spill_insert_kernel(const uint2* __restrict__ spill, const uint32_t* __restrict__ nspill,
                    unsigned long long* slot, uint32_t npairs, uint32_t pp, uint32_t g, uint32_t* __restrict__ mark,
                    uint2* __restrict__ rank) {
  const uint32_t n = *nspill;
  for (uint64_t i0 = ((uint64_t)blockIdx.x * 256 + threadIdx.x) & ~31ull; i0 < n; i0 += (uint64_t)gridDim.x * 256) {
    const uint64_t i = i0 + (threadIdx.x & 31u);
    const bool ok[1] = {i < n};
    const uint2 r = ok[0] ? __ldg(spill + i) : make_uint2(0u, 0u);
    const int32_t key[1] = {(int32_t)r.x};
    const uint32_t hv[1] = {ej_hash32(r.y)};
    uint32_t q = ((hv[0] >> (32u - MSD_BUCKET_BITS + g)) + 1u) * pp;  // pair behind the group
    for (bool found = !ok[0]; !found;) {  // ends: more than half of the slots stay empty
      uint4 w[4];
#pragma unroll
      for (uint32_t e = 0; e < 4; e++) {
        const uint32_t a = q + e < npairs ? q + e : q + e - npairs;
        w[e] = __ldcg(reinterpret_cast<const uint4*>(slot) + a);
      }
#pragma unroll
      for (uint32_t e = 0; e < 4; e++) {
        const uint32_t y = hv[0] << 1 | 1u;
        found = found || (w[e].x | w[e].y) == 0u || (w[e].z | w[e].w) == 0u || (w[e].y | 1u) == y || (w[e].w | 1u) == y;
        if (!found) q++;
      }
      if (q >= npairs) q -= npairs;
    }
    const uint32_t at[1] = {q < npairs ? q : q - npairs};
    EjSlotMark m[1];
    ej_slot_insert<1, true>(slot, npairs, key, hv, ok, m, at);
    if (ok[0]) {
      mark[i] = m[0].mark;
      rank[i] = make_uint2(m[0].rank, (uint32_t)m[0].first);
    }
  }
}

__global__ void __launch_bounds__(256)
spill_reserve_kernel(const uint2* __restrict__ spill, const uint32_t* __restrict__ nspill, uint2* __restrict__ slot,
                     const uint32_t* __restrict__ mark, const uint2* __restrict__ rank, uint32_t g,
                     int32_t* __restrict__ rkey, uint32_t* __restrict__ gcursor) {
  const uint32_t n = *nspill;
  for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (uint64_t)gridDim.x * 256) {
    const uint32_t m = __ldg(mark + i);
    const uint2 r = __ldg(rank + i);
    if (!m || !(r.x & EJ_SLOT_OPENER)) continue;
    const uint32_t c = slot[m - 1u].x;
    uint32_t lo = atomicAdd(gcursor + (ej_hash32(__ldg(&spill[i].y)) >> (32u - MSD_BUCKET_BITS + g)),
                            c + (c >= 31u ? 1u : 0u));
    if (c >= 31u) rkey[lo++] = (int32_t)c;
    if (r.x & 1u) rkey[lo] = (int32_t)r.y;
    slot[m - 1u].x = lo << 5 | min(c, 31u);
  }
}

__global__ void __launch_bounds__(256)
spill_place_kernel(const uint2* __restrict__ spill, const uint32_t* __restrict__ nspill, const uint2* __restrict__ slot,
                   const uint32_t* __restrict__ mark, const uint2* __restrict__ rank, int32_t* __restrict__ rkey) {
  const uint32_t n = *nspill;
  for (uint64_t i = (uint64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (uint64_t)gridDim.x * 256) {
    const uint32_t m = __ldg(mark + i);
    if (m) rkey[(__ldg(&slot[m - 1u].x) >> 5) + (__ldg(&rank[i].x) & ~EJ_SLOT_OPENER)] = (int32_t)__ldg(&spill[i].x);
  }
}

// bucket groups of 2^g buckets of about LS_ROWS rows in all
uint32_t msd_group_bits(uint64_t n) {
  uint32_t g = 0;
  while (g < LS_MAX_GROUP_BITS && ((uint64_t)LS_ROWS << MSD_BUCKET_BITS) >= (n << (g + 1))) g++;
  return g;
}

}  // namespace

void ej_msd_plan_add(ej_plan_bytes& p, ej_msd_plan& mp, uint64_t n) {
  mp.n = n;
  ej_radix_plan_add(p, mp.pass1, n);
  // the second pass: at most one partial tile more per segment
  mp.pass2.n = n;
  mp.pass2.ntiles = ej_radix_tiles(n) + 256;
  const uint64_t cells = (uint64_t)mp.pass2.ntiles * 256;
  mp.pass2.hist_off = p.add(cells * sizeof(uint32_t));
  mp.pass2.offs_off = p.add((cells + 1) * sizeof(uint32_t));
  mp.pass2.scan_off = p.add(ej_scan_scratch_bytes(cells));
  mp.desc_off = p.add((size_t)mp.pass2.ntiles * sizeof(ej_rx_tile));
  mp.seg_off = p.add(sizeof(MsdSegments));
  mp.bstart_off = p.add((MSD_BUCKETS + 1) * sizeof(uint32_t));
}

uint32_t ej_msd_slot_pairs(uint64_t n) {
  const uint64_t groups = MSD_BUCKETS >> msd_group_bits(n);
  return (uint32_t)((n + groups) / groups * groups);  // above n, the same for every group
}

// the two radix passes (rows in tmp_b, tmp_a free again) and the bucket bounds
static ej_status msd_passes(ej_handle* h, const ej_msd_plan& mp, const ej_tuple* R, ej_tuple* tmp_a, ej_tuple* tmp_b,
                            uint32_t** bounds, uint32_t* gave_up = nullptr) {
  // 1. by bits 24..31
  ej_radix_plan p1 = mp.pass1;
  p1.gave_up = gave_up;
  EJ_TRY(ej_partition_pass(h, p1, R, tmp_a, 24u, 8u, EJ_DIGIT_HASH));
  // 2. by bits 16..23 inside every segment, tiles laid out on the device
  MsdSegments* seg = reinterpret_cast<MsdSegments*>(ej_arena_at(h, mp.seg_off));
  ej_rx_tile* desc = reinterpret_cast<ej_rx_tile*>(ej_arena_at(h, mp.desc_off));
  const uint32_t* offs1 = reinterpret_cast<const uint32_t*>(ej_arena_at(h, mp.pass1.offs_off));
  msd_segments_kernel<<<1, 256, 0, h->stream>>>(offs1, mp.pass1.ntiles, mp.n, seg);
  EJ_TRY(ej_check_launch(h, "msd_segments_kernel"));
  msd_tiles_kernel<<<(mp.pass2.ntiles + 255) / 256, 256, 0, h->stream>>>(seg, desc, mp.pass2.ntiles);
  EJ_TRY(ej_check_launch(h, "msd_tiles_kernel"));
  ej_radix_plan p2 = mp.pass2;
  p2.tiles = desc;
  p2.gave_up = gave_up;
  EJ_TRY(ej_partition_pass(h, p2, tmp_a, tmp_b, 16u, 8u, EJ_DIGIT_HASH));
  // 3. bucket bounds
  uint32_t* bstart = reinterpret_cast<uint32_t*>(ej_arena_at(h, mp.bstart_off));
  const uint32_t* offs2 = reinterpret_cast<const uint32_t*>(ej_arena_at(h, mp.pass2.offs_off));
  msd_bucket_kernel<<<(MSD_BUCKETS + 1 + 255) / 256, 256, 0, h->stream>>>(seg, offs2, mp.n, bstart);
  EJ_TRY(ej_check_launch(h, "msd_bucket_kernel"));
  *bounds = bstart;
  return EJ_OK;
}

ej_status ej_msd_slots(ej_handle* h, const ej_msd_plan& mp, const ej_tuple* R, ej_tuple* tmp_a, ej_tuple* tmp_b,
                       uint4* pair, uint32_t npairs, int32_t* rkey, uint32_t* gcursor, uint32_t* mark,
                       uint32_t* nspill, uint32_t* gave_up) {
  uint32_t* bstart = nullptr;
  EJ_TRY(msd_passes(h, mp, R, tmp_a, tmp_b, &bstart, gave_up));
  const uint32_t g = msd_group_bits(mp.n), groups = MSD_BUCKETS >> g, pp = npairs / groups;
  const int smem = (int)(2u * pp * sizeof(unsigned long long));
  // 32 KB and less (LS_ROWS rows a group or fewer): within the default limit, which
  // is the function's, for every handle and thread, so it is left alone
  if (smem > 48 * 1024 - 256) return ej_fail(h, EJ_ERR_INTERNAL, "bucket group of %u pairs", pp);
  uint2* spill = reinterpret_cast<uint2*>(tmp_a);
  msd_slots_kernel<<<groups, LS_THREADS, smem, h->stream>>>(tmp_b, bstart, g, npairs, pp, pair, rkey, gcursor, spill,
                                                           nspill, mark, gave_up);
  EJ_TRY(ej_check_launch(h, "msd_slots_kernel"));
  // the spilled rows' marks (mark held large groups' ranks before); their ranks
  // in tmp_b, whose rows are in the table now
  uint2* rank = reinterpret_cast<uint2*>(tmp_b);
  uint2* slot = reinterpret_cast<uint2*>(pair);
  const unsigned blocks = (unsigned)h->num_sms * 2;
  spill_insert_kernel<<<blocks, 256, 0, h->stream>>>(spill, nspill, reinterpret_cast<unsigned long long*>(pair), npairs,
                                                    pp, g, mark, rank);
  EJ_TRY(ej_check_launch(h, "spill_insert_kernel"));
  spill_reserve_kernel<<<blocks, 256, 0, h->stream>>>(spill, nspill, slot, mark, rank, g, rkey, gcursor);
  EJ_TRY(ej_check_launch(h, "spill_reserve_kernel"));
  spill_place_kernel<<<blocks, 256, 0, h->stream>>>(spill, nspill, slot, mark, rank, rkey);
  return ej_check_launch(h, "spill_place_kernel");
}

ej_status ej_msd_sort(ej_handle* h, const ej_msd_plan& mp, const ej_tuple* R, ej_tuple* tmp_a, ej_tuple* tmp_b,
                      int32_t* rkey, int32_t* rval) {
  if (mp.n == 0) return EJ_OK;
  if (mp.n >= 0xFFFFFFFFull) return ej_fail(h, EJ_ERR_TOO_LARGE, "table of %llu rows", (unsigned long long)mp.n);
  uint32_t* bstart = nullptr;
  EJ_TRY(msd_passes(h, mp, R, tmp_a, tmp_b, &bstart));
  // every bucket by bits 0..15 into the columns
  const uint32_t g = msd_group_bits(mp.n);
  EJ_CUDA(h, cudaFuncSetAttribute(msd_local_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LsSmem)));
  msd_local_kernel<<<MSD_BUCKETS >> g, LS_THREADS, sizeof(LsSmem), h->stream>>>(tmp_b, tmp_a, bstart, g, rkey, rval);
  return ej_check_launch(h, "msd_local_kernel");
}
