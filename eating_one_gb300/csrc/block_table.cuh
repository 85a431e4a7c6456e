// block_table.cuh - a hash table of up to 16384 R rows in one CTA's shared
// memory (device code), shared by the block nested loop (bnlj.cu) and the joins
// whose whole build side fits (small_join.cu).
//
// Rows are grouped by bucket (top hash bits, about one row a bucket or less)
// by a counting sort, in two columns, with 2-byte bucket starts.  A warp
// looks its tuples up together and collects the matches in a shared-memory
// buffer that becomes rows with one atomic add on the output cursor and
// coalesced stores.  The buffers share their memory with the build's bucket
// counters.
#pragma once

#include "ej_device.cuh"

constexpr uint32_t BT_ROWS = 16384;       // 128 KB of columns, 32 KB of starts, 64 KB of counters
constexpr uint32_t BT_MIN_BUCKETS = 256;  // a multiple of 32 buckets per warp of the scan
constexpr uint32_t BT_BUF = 128;          // matches a warp collects
constexpr uint32_t BT_DEEP = 128;         // buckets of more rows are searched by the whole warp
constexpr uint32_t BT_MANY = 16;          // matches of a tuple whose rows the whole warp writes

struct BtTable {
  int32_t* rval;       // [n] the rows, bucket by bucket
  int32_t* rkey;       // [n]
  uint32_t* count;     // [2^lg] the build's bucket counters
  uint16_t* start;     // [2^lg + 1] first row of each bucket, then the end
  uint32_t* scan_tmp;  // [warps]
  uint32_t lg;
};

__device__ __forceinline__ uint32_t bt_bucket(int32_t v, uint32_t lg) { return ej_hash32((uint32_t)v) >> (32u - lg); }

// The table of R[0, n), 2^lg >= n buckets, 2^lg a multiple of 32 per warp.
// The rows are read twice (they sit in L2), so that none waits in registers.
// Returns whether some bucket is deep (more than BT_DEEP rows).
template <int THREADS>
__device__ __forceinline__ bool bt_build(const BtTable& t, const int2* __restrict__ R, uint32_t n) {
  constexpr uint32_t WARPS = THREADS / 32;
  const uint32_t nb = 1u << t.lg;
  for (uint32_t b = threadIdx.x; b < nb; b += THREADS) t.count[b] = 0u;
  __syncthreads();
#pragma unroll 8
  for (uint32_t i = threadIdx.x; i < n; i += THREADS) atomicAdd(&t.count[bt_bucket(__ldg(&R[i].y), t.lg)], 1u);
  __syncthreads();
  // exclusive scan of the counts: each warp a contiguous share, 32 buckets a
  // step, then the warps' totals; the counters become row cursors
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t share = nb / WARPS, b0 = warp * share;
  uint32_t run = 0;
  for (uint32_t b = b0 + lane; b < b0 + share; b += 32) run += t.count[b];
  run = __reduce_add_sync(EJ_FULL_MASK, run);
  if (lane == 0) t.scan_tmp[warp] = run;
  __syncthreads();
  run = __reduce_add_sync(EJ_FULL_MASK, lane < warp ? t.scan_tmp[lane] : 0u);
  bool deep = false;
  for (uint32_t b = b0 + lane; b < b0 + share; b += 32) {
    const uint32_t c = t.count[b];
    deep |= c > BT_DEEP;
    const uint32_t incl = ej_warp_inclusive_sum(c);
    t.count[b] = run + incl - c;
    t.start[b] = (uint16_t)(run + incl - c);
    run += __shfl_sync(EJ_FULL_MASK, incl, 31);
  }
  if (threadIdx.x == 0) t.start[nb] = (uint16_t)n;
  __syncthreads();
#pragma unroll 8
  for (uint32_t i = threadIdx.x; i < n; i += THREADS) {
    const int2 r = __ldg(R + i);
    const uint32_t pos = atomicAdd(&t.count[bt_bucket(r.y, t.lg)], 1u);
    t.rval[pos] = r.y;
    t.rkey[pos] = r.x;
  }
  return __syncthreads_or(deep) != 0;
}

// the output of a join: rows past cap are dropped, the cursor counts them all
struct BtOut {
  ej_result* rows;
  uint64_t cap;
  unsigned long long* cursor;
  ej_dev_status* st;  // records EJ_ERR_CAPACITY when not null
  __device__ __forceinline__ unsigned long long reserve(uint32_t n) const {
    unsigned long long off = 0;
    if ((threadIdx.x & 31u) == 0) {
      off = atomicAdd(cursor, (unsigned long long)n);
      if (st && off <= cap && off + n > cap) ej_set_status(st, EJ_ERR_CAPACITY, 0u);
    }
    return __shfl_sync(EJ_FULL_MASK, off, 0);
  }
  __device__ __forceinline__ void put(unsigned long long pos, int32_t rkey, int32_t rval, int2 s) const {
    if (pos < cap) __stcs(reinterpret_cast<int4*>(rows + pos), make_int4(rkey, rval, s.x, s.y));
  }
};

constexpr int BT_NULL = -1;  // the position of a NULL-extended row

// A warp's collected matches: {S key, R position}, or with S (the relation)
// {S row, R position}, which NULL-extended rows need.
struct BtBuffer {
  int2* e;
  uint32_t held;
};

template <bool INDEXED>
__device__ __forceinline__ void bt_flush(const BtTable& t, BtBuffer& f, const int2* __restrict__ S, const BtOut& o) {
  __syncwarp();
  const unsigned long long off = o.reserve(f.held);
  for (uint32_t k = threadIdx.x & 31u; k < f.held; k += 32) {
    const int2 e = f.e[k];
    const bool null = INDEXED && e.y == BT_NULL;
    const int32_t v = null ? EJ_NULL_KEY : t.rval[e.y];
    const int2 s = INDEXED ? __ldg(S + (uint32_t)e.x) : make_int2(e.x, v);
    o.put(off + k, null ? EJ_NULL_KEY : t.rkey[e.y], v, s);
  }
  __syncwarp();
  f.held = 0;
}

// The rows of bucket [at, at + n) with val v, searched by the whole warp: their
// number, and the last one's position in *last (in every lane)
__device__ __forceinline__ uint32_t bt_count_deep(const BtTable& t, uint32_t at, uint32_t n, int32_t v,
                                                  uint32_t* last) {
  uint32_t c = 0, l = 0;
  for (uint32_t k = threadIdx.x & 31u; k < n; k += 32)
    if (t.rval[at + k] == v) {
      c++;
      l = at + k;
    }
  *last = __reduce_max_sync(EJ_FULL_MASK, l);
  return __reduce_add_sync(EJ_FULL_MASK, c);
}

// ... joined with the S tuple s, written by the whole warp from out[pos] on
__device__ __forceinline__ void bt_write_many(const BtTable& t, int2 s, unsigned long long pos, const BtOut& o) {
  const uint32_t b = bt_bucket(s.y, t.lg), end = t.start[b + 1];
  for (uint32_t k0 = t.start[b]; k0 < end; k0 += 32) {
    const uint32_t k = k0 + (threadIdx.x & 31u);
    const bool hit = k < end && t.rval[k] == s.y;
    const unsigned hits = __ballot_sync(EJ_FULL_MASK, hit);
    if (hit) o.put(pos + __popc(hits & ej_lanemask_lt()), t.rkey[k], s.y, s);
    pos += __popc(hits);
  }
}

// Looks up the warp's 32 * N tuples s (ok: a tuple is there; INDEXED: tuple j
// of the lane is S[row0 + 32 j + lane]); OUTER: one NULL-extended row for a
// tuple without a match (needs INDEXED).  All buckets are walked together, one
// row a round, but for deep ones, which the warp searches together, once for
// tuples of one val; matches collect in f.  A step with more than the buffer holds
// writes its rows itself: the warp together those of a tuple with BT_MANY matches
// or more, else each lane its own.  (Lanes that each write a run store to 32 lines
// at once.  2^20 S rows, half of them with 128 matches, 16384 R rows: 1.26 ms, by
// warp 0.45, tables in global memory 0.49.  8000 rows of one key that a hundredth
// of 2^20 S rows hit: 11.6, 0.45 and 4.1 ms.)  COUNT_ONLY: returns the lane's
// matches.  DEEP: some bucket is (told once per table).
template <bool DEEP, bool COUNT_ONLY, bool OUTER, bool INDEXED, int N>
__device__ __forceinline__ uint32_t bt_probe(const BtTable& t, const int2 (&s)[N], const bool (&ok)[N], uint32_t row0,
                                             const int2* __restrict__ S, BtBuffer& f, const BtOut& o) {
  static_assert(!OUTER || INDEXED, "NULL-extended rows are collected by S row");
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t at[N], rows[N], c[N], hit[N], deepest = 0, mine = 0;
#pragma unroll
  for (int j = 0; j < N; j++) {
    const uint32_t b = bt_bucket(s[j].y, t.lg);
    at[j] = ok[j] ? t.start[b] : 0u;
    rows[j] = ok[j] ? t.start[b + 1] - at[j] : 0u;
    c[j] = hit[j] = 0;
    deepest = max(deepest, rows[j]);
  }
  if (DEEP && __any_sync(EJ_FULL_MASK, deepest > BT_DEEP)) {
    deepest = 0;
#pragma unroll
    for (int j = 0; j < N; j++) {
      for (unsigned m = __ballot_sync(EJ_FULL_MASK, rows[j] > BT_DEEP); m;) {
        const int leader = __ffs(m) - 1;
        const int32_t v = __shfl_sync(EJ_FULL_MASK, s[j].y, leader);
        uint32_t last;
        const uint32_t n = bt_count_deep(t, __shfl_sync(EJ_FULL_MASK, at[j], leader),
                                         __shfl_sync(EJ_FULL_MASK, rows[j], leader), v, &last);
        const bool same = (m >> lane & 1u) && s[j].y == v;
        if (same) {
          c[j] = n;
          hit[j] = last;
          rows[j] = 0;  // done
        }
        m &= ~__ballot_sync(EJ_FULL_MASK, same);
      }
      deepest = max(deepest, rows[j]);
    }
  }
  for (uint32_t k = 0; k < deepest; k++) {
#pragma unroll
    for (int j = 0; j < N; j++)
      if (k < rows[j] && t.rval[at[j] + k] == s[j].y) {
        c[j]++;
        hit[j] = at[j] + k;
      }
  }
#pragma unroll
  for (int j = 0; j < N; j++) {
    if (OUTER && ok[j] && c[j] == 0) {
      c[j] = 1;
      hit[j] = (uint32_t)BT_NULL;
    }
    mine += c[j];
  }
  if (COUNT_ONLY) return mine;
  if (!__any_sync(EJ_FULL_MASK, mine != 0)) return 0;
  const uint32_t incl = ej_warp_inclusive_sum(mine);
  const uint32_t total = __shfl_sync(EJ_FULL_MASK, incl, 31);
  if (f.held + total > BT_BUF && f.held) bt_flush<INDEXED>(t, f, S, o);
  if (total > BT_BUF) {  // more than the buffer holds
    unsigned long long pos = o.reserve(total) + (incl - mine);
#pragma unroll
    for (int j = 0; j < N; j++) {
      for (unsigned m = __ballot_sync(EJ_FULL_MASK, c[j] >= BT_MANY); m; m &= m - 1u) {
        const int src = __ffs(m) - 1;
        const int2 tuple = make_int2(__shfl_sync(EJ_FULL_MASK, s[j].x, src), __shfl_sync(EJ_FULL_MASK, s[j].y, src));
        bt_write_many(t, tuple, __shfl_sync(EJ_FULL_MASK, pos, src), o);
      }
      if (c[j] >= BT_MANY) pos += c[j];
      uint32_t i = hit[j];  // the last match, then those before it
      for (uint32_t left = c[j] >= BT_MANY ? 0u : c[j]; left != 0; pos++) {
        const bool null = OUTER && i == (uint32_t)BT_NULL;
        o.put(pos, null ? EJ_NULL_KEY : t.rkey[i], null ? EJ_NULL_KEY : s[j].y, s[j]);
        if (--left)
          do i--;
          while (t.rval[i] != s[j].y);
      }
    }
    return 0;
  }
  uint32_t pos = f.held + incl - mine;
  f.held += total;
#pragma unroll
  for (int j = 0; j < N; j++) {
    uint32_t i = hit[j];
    for (uint32_t left = c[j]; left != 0; pos++) {
      f.e[pos] = make_int2(INDEXED ? (int)(row0 + 32u * j + lane) : s[j].x, (int)i);
      if (--left)
        do i--;
        while (t.rval[i] != s[j].y);
    }
  }
  return 0;
}
