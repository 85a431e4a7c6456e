// slot_table.cuh - hash tables by open addressing (device code): the build's
// steps and the probe's find, shared by the single joins (hash_join.cu), the
// star join (index.cu), the batched joins (batch.cu) and, for the rows that its
// bucket groups spill, the build of large tables (msd.cu).
//
// A table of n rows has one 8-byte slot {x, y} per distinct key, in an array of
// npairs >= n aligned pairs (so at most half full), found from the key's home
// pair mulhi(hash32(val), npairs) by walking on, pair by pair, to the key or to
// a pair with an empty slot:
//   one row         {key, hash << 1}
//   several rows    {lo << 5 | min(rows, 31), hash << 1 | 1}: their keys are
//                   rkey[lo ...]; from 31 rows on their number is rkey[lo - 1]
//   none            {0, 0}
// The hash is a bijection of val, so an equal hash is an equal val; its top bit,
// which the shift drops, is told by the slot's place: hashes that differ only
// there have homes npairs / 2 apart, and a walk is shorter (it crosses full
// pairs only, of which n rows fill fewer than npairs / 2).  One row whose slot
// would be all zeros (key 0, hash << 1 = 0) takes the several-rows form.
// A probe of a present or an absent key is answered by one 16-byte load of its
// home pair unless the pair is full of other keys (under 2% of the probes at a
// quarter load, a tenth at half), and for a single row the load brings its key.
//
// Build, without sorting: every row claims an empty slot for its key with one
// compare-and-swap that already writes the final single-row form, so a table of
// unique keys is done after one pass; a row that finds its key (or meets it in
// its warp) turns the slot into a counter, or counts itself in, and is marked
// with its rank.  When there are any, two more passes reserve the runs and
// place the marked rows.  Rows of one key in a warp go together, so that a key
// with very many rows costs 1/32 of the atomics.
//
// What bounds it: the build, the round trips of its compare-and-swaps (40 to 60 G
// rows/s; the L2 takes 75 to 115 G random ones/s while the slots fit it); the
// probe, its gathers' L2 round trips and, with runs of several rows, the run
// keys' gathers.  One GB300, |S| = 4 |R|, a tenth of S absent,
// build and one-pass probe in us, this table and the hash-sorted one it replaced
// (MSD passes, bucket sort, bucket bounds), then the whole call into a given
// output: 2^18 rows 32 + 17 and 80 + 25 (89, 152); 2^20 50 + 45 and 94 + 73 (136,
// 213).  Above 2^21 rows (built by groups, msd.cu) the whole call: 3 M 322 and 349;
// 3 M rows of 1 M keys 425 and 454; 3 M of 375 K 575 and 663; 12 M 1075 and 1325;
// 12 M of 4 M keys 1437 and 1524; 2^25 2711 and 3475.  Tried and
// dropped on the way: buckets by hash with the row in the slot when alone, else a
// pointer to the bucket's rows - unsorted rows walked by each probe (2^20 151, but
// 3 M of 375 K 975), rows grouped by key in a further pass (180 and 660): the
// buckets that two keys share cost every warp a second walk.
#pragma once

#include "ej_device.cuh"
#include "probe_write.cuh"

struct EjSlotTable {
  const uint4* pair;    // [npairs]
  const int32_t* rkey;  // runs of the keys with several rows
  uint32_t npairs;
  uint32_t run_words;   // words of rkey
};

__device__ __forceinline__ EjSlotTable ej_slots_of(const ej_table_view& t) { return {t.pair, t.rkey, t.npairs, t.run_words}; }

__device__ __forceinline__ uint32_t ej_home_pair(uint32_t hash, uint32_t npairs) { return __umulhi(hash, npairs); }

// ---- build ----------------------------------------------------------------------

// The slot after `at` on a key's walk: in each pair first the slot that the lowest
// bit of the hash names, then the other.  (All keys beginning with a pair's first
// slot found it taken almost twice as often.)
__device__ __forceinline__ uint32_t ej_next_slot(uint32_t at, uint32_t hash, uint32_t npairs) {
  if (((at ^ hash) & 1u) == 0u) return at ^ 1u;
  const uint32_t pair = (at >> 1) + 1u;
  return 2u * (pair == npairs ? 0u : pair) + (hash & 1u);
}

// A row of a key with several: mark = 1 + its key's slot (0: not one of them),
// rank = its rank among the key's rows.  The row that turned the slot's single-
// row form into a counter has rank 1, EJ_SLOT_OPENER set, and keeps the slot's
// former key in `first`; so does, with rank 0 and no first, the first row of a
// slot that began as a counter.
struct EjSlotMark {
  uint32_t mark, rank;
  int32_t first;
};
constexpr uint32_t EJ_SLOT_OPENER = 0x80000000u;

// N rows of this lane (ok[j]: there is one) claim slots of the zeroed array or
// are marked.  All lanes' walks advance together, one compare-and-swap per row
// and round.  FROM: the walks begin at pair from[j], instead of the home, from
// which the key's walk leads there over full pairs.
template <int N, bool FROM = false>
__device__ __forceinline__ void ej_slot_insert(unsigned long long* __restrict__ slot, uint32_t npairs,
                                               const int32_t (&key)[N], const uint32_t (&hash)[N],
                                               const bool (&ok)[N], EjSlotMark (&m)[N],
                                               const uint32_t* from = nullptr) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t walk = 0, alone = 0, peers[N], at[N];
#pragma unroll
  for (int j = 0; j < N; j++) {
    peers[j] = __match_any_sync(EJ_FULL_MASK, hash[j]) & __ballot_sync(EJ_FULL_MASK, ok[j]);
    at[j] = 2u * (FROM ? from[j] : ej_home_pair(hash[j], npairs)) + (hash[j] & 1u);
    m[j] = {0u, 0u, 0};
    if (ok[j] && __ffs(peers[j]) - 1 == (int)lane) walk |= 1u << j;  // the first of the key's rows in the warp
  }
  while (walk) {  // ends: more than half of the slots stay empty, and a slot changes form once
    unsigned long long old[N];
#pragma unroll
    for (int j = 0; j < N; j++)
      if (walk >> j & 1u) {
        // the final form, or a counter: of several rows in this warp, or of a
        // row whose final form would be all zeros
        const uint32_t y = hash[j] << 1, n = __popc(peers[j]);
        old[j] = atomicCAS(slot + at[j], 0ull,
                           n == 1u && (y | (uint32_t)key[j]) ? (unsigned long long)y << 32 | (uint32_t)key[j]
                                                             : (unsigned long long)(y | 1u) << 32 | n);
      }
#pragma unroll
    for (int j = 0; j < N; j++) {
      if (!(walk >> j & 1u)) continue;
      const uint32_t y = hash[j] << 1, n = __popc(peers[j]);
      unsigned long long w = old[j];
      if (w == 0ull) {
        walk &= ~(1u << j);
        if (n == 1u && (y | (uint32_t)key[j])) alone |= 1u << j; else m[j].rank = EJ_SLOT_OPENER;
      } else if (((uint32_t)(w >> 32) | 1u) != (y | 1u)) {
        at[j] = ej_next_slot(at[j], hash[j], npairs);
      } else {
        walk &= ~(1u << j);
        if (!(w >> 32 & 1u)) {  // the single-row form: make it a counter, unless another row just did
          const unsigned long long seen =
              atomicCAS(slot + at[j], w, (unsigned long long)(y | 1u) << 32 | (1u + n));
          if (seen == w) {
            m[j].rank = EJ_SLOT_OPENER | 1u;
            m[j].first = (int32_t)(uint32_t)w;
            continue;
          }
        }
        m[j].rank = atomicAdd(reinterpret_cast<uint32_t*>(slot + at[j]), n);
      }
    }
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < N; j++) {
    const int leader = peers[j] ? __ffs(peers[j]) - 1 : 0;
    const uint32_t s = __shfl_sync(EJ_FULL_MASK, at[j], leader);
    const uint32_t rank = __shfl_sync(EJ_FULL_MASK, m[j].rank, leader);
    if (!ok[j] || (alone >> j & 1u)) continue;
    m[j].mark = 1u + s;
    if ((int)lane != leader) m[j].rank = (rank & ~EJ_SLOT_OPENER) + __popc(peers[j] & ej_lanemask_lt());
  }
}

// The final slots of keys with several rows, by the rows that opened their
// counters (open[j]; rank as marked): reserves the runs on *cursor.
template <int N>
__device__ __forceinline__ void ej_slot_reserve(uint2* __restrict__ slot, const uint32_t (&mark)[N],
                                                const uint2 (&rank)[N], int32_t* __restrict__ rkey,
                                                uint32_t* __restrict__ cursor) {
  uint32_t c[N], mine = 0;
#pragma unroll
  for (int j = 0; j < N; j++) c[j] = mark[j] && (rank[j].x & EJ_SLOT_OPENER) ? slot[mark[j] - 1u].x : 0u;
#pragma unroll
  for (int j = 0; j < N; j++) mine += c[j] + (c[j] >= 31u ? 1u : 0u);
  if (!__any_sync(EJ_FULL_MASK, mine != 0u)) return;
  const uint32_t incl = ej_warp_inclusive_sum(mine);
  uint32_t lo = 0;
  if ((threadIdx.x & 31u) == 31u) lo = atomicAdd(cursor, incl);
  lo = __shfl_sync(EJ_FULL_MASK, lo, 31) + incl - mine;
#pragma unroll
  for (int j = 0; j < N; j++) {
    if (!c[j]) continue;
    if (c[j] >= 31u) rkey[lo++] = (int32_t)c[j];
    if (rank[j].x & 1u) rkey[lo] = (int32_t)rank[j].y;
    slot[mark[j] - 1u].x = lo << 5 | min(c[j], 31u);
    lo += c[j];
  }
}

// ---- probe ----------------------------------------------------------------------

__device__ __forceinline__ bool ej_pair_full(const uint4& q) { return (q.x | q.y) != 0u && (q.z | q.w) != 0u; }

// Rows of the run of 31 rows and more that begins at rkey[lo].  Never past the
// array, also when a scan of the build's passes gave up waiting (the call then
// reports it) and bucket groups wrote over each other's runs.
__device__ __forceinline__ uint32_t ej_run_length(const int32_t* rkey, uint32_t lo, uint32_t run_words) {
  return min((uint32_t)__ldg(rkey + lo - 1), run_words - lo);
}

// The matches of N probe values (ok[j] false: none): c[j] rows, the first at
// rkey[lo[j]], or lo[j] = INLINE_RUN and c[j] = 1: the row with key key[j].
template <int N>
__device__ __forceinline__ void ej_slot_find(const EjSlotTable& t, const int32_t (&v)[N], const bool (&ok)[N],
                                             uint32_t (&lo)[N], uint32_t (&c)[N], int32_t (&key)[N]) {
  uint32_t h2[N], p[N], walk = 0;
  uint4 q[N];
#pragma unroll
  for (int j = 0; j < N; j++) {
    const uint32_t hv = ej_hash32((uint32_t)v[j]);
    h2[j] = hv << 1 | 1u;
    p[j] = ej_home_pair(hv, t.npairs);
    q[j] = make_uint4(0u, 0u, 0u, 0u);
    if (ok[j]) q[j] = __ldg(t.pair + p[j]);
  }
#pragma unroll
  for (int j = 0; j < N; j++)
    if (ej_pair_full(q[j]) && (q[j].y | 1u) != h2[j] && (q[j].w | 1u) != h2[j]) walk |= 1u << j;
  while (walk) {  // the pairs were full of other keys
#pragma unroll
    for (int j = 0; j < N; j++)
      if (walk >> j & 1u) {
        p[j] = p[j] + 1u == t.npairs ? 0u : p[j] + 1u;
        q[j] = __ldg(t.pair + p[j]);
      }
#pragma unroll
    for (int j = 0; j < N; j++)
      if ((walk >> j & 1u) && (!ej_pair_full(q[j]) || (q[j].y | 1u) == h2[j] || (q[j].w | 1u) == h2[j]))
        walk &= ~(1u << j);
  }
  uint32_t longest = 0;
#pragma unroll
  for (int j = 0; j < N; j++) {
    // an empty slot can only look like a key whose hash << 1 is zero
    const bool second = (q[j].w | 1u) == h2[j] && (q[j].z | q[j].w) != 0u;
    const uint32_t x = second ? q[j].z : q[j].x, y = second ? q[j].w : q[j].y;
    const bool run = y == h2[j], one = (y ^ 1u) == h2[j] && (x | y) != 0u;
    key[j] = (int32_t)x;
    lo[j] = run ? x >> 5 : INLINE_RUN;
    c[j] = run ? x & 31u : one ? 1u : 0u;
    longest = max(longest, c[j]);
  }
  if (longest == 31u) {
#pragma unroll
    for (int j = 0; j < N; j++)
      if (c[j] == 31u) c[j] = ej_run_length(t.rkey, lo[j], t.run_words);
  }
}

// probes [base, min(base + 128, nP)): tuples and matches (OUTER: an unmatched
// probe gets one row, marked by lo = NULL_RUN)
template <bool OUTER>
__device__ __forceinline__ void ej_slot_probe(const ej_tuple* __restrict__ P, uint64_t base, uint64_t nP,
                                              const EjSlotTable& t, EjProbeWarp& w, int32_t (&key)[PR_ITEMS]) {
  const unsigned lane = threadIdx.x & 31u;
  int32_t v[PR_ITEMS];
  bool ok[PR_ITEMS];
#pragma unroll
  for (int j = 0; j < PR_ITEMS; j++) {
    const uint64_t idx = base + (uint64_t)j * 32 + lane;
    ok[j] = idx < nP;
    w.s[j] = ok[j] ? __ldcs(reinterpret_cast<const int2*>(P) + idx) : make_int2(0, 0);
    v[j] = w.s[j].y;
  }
  ej_slot_find<PR_ITEMS>(t, v, ok, w.lo, w.cnt, key);
  if (OUTER) {
#pragma unroll
    for (int j = 0; j < PR_ITEMS; j++)
      if (ok[j] && w.cnt[j] == 0) {
        w.cnt[j] = 1;
        w.lo[j] = NULL_RUN;
      }
  }
}

// The rows of a warp tile with runs, from out[off] on: a function of its own, so
// that its registers (the run keys) do not burden the tiles without.  Its
// arguments travel in registers (a structure passed by reference would live in
// local memory: 1242 us instead of 1098 for the one-pass probes of 2^24 rows of
// four a key).
static __device__ __noinline__ void ej_slot_emit_runs(int4 skey, int4 sval, uint4 lo, uint4 cnt, int4 key4,
                                                      const int32_t* __restrict__ rkey, unsigned long long off,
                                                      ej_result* __restrict__ out, uint64_t cap, int4* stage) {
  const EjProbeWarp p = {{make_int2(skey.x, sval.x), make_int2(skey.y, sval.y), make_int2(skey.z, sval.z),
                          make_int2(skey.w, sval.w)},
                         {lo.x, lo.y, lo.z, lo.w},
                         {cnt.x, cnt.y, cnt.z, cnt.w}};
  const int32_t key[PR_ITEMS] = {key4.x, key4.y, key4.z, key4.w};
  ej_table_view t;
  t.rkey = rkey;
  int32_t kk[PR_ITEMS][PW_PREFETCH];
  ej_probe_prefetch<EJ_KEYS_WINDOW, true>(t, p, kk, key);
  ej_emit_warp<true>(p, kk, t, off, out, cap, stage);
}

// The rows of a warp tile from out[off] on.  Tiles with at most one match per
// probe, all of them from slots (unique keys, an outer join's NULL-extended
// rows), go straight out in lane order; the others as runs.
__device__ __forceinline__ void ej_slot_emit(const EjProbeWarp& p, const int32_t (&key)[PR_ITEMS],
                                             const ej_table_view& t, unsigned long long off,
                                             ej_result* __restrict__ out, uint64_t cap, int4* stage) {
  bool one = true;
#pragma unroll
  for (int j = 0; j < PR_ITEMS; j++) one &= p.cnt[j] == 0u || p.lo[j] >= INLINE_RUN;
  if (__all_sync(EJ_FULL_MASK, one)) {
    const unsigned lt = ej_lanemask_lt();
#pragma unroll
    for (int j = 0; j < PR_ITEMS; j++) {
      const unsigned b = __ballot_sync(EJ_FULL_MASK, p.cnt[j] != 0u);
      const unsigned long long pos = off + (unsigned)__popc(b & lt);
      const bool null = p.lo[j] == NULL_RUN;
      if (p.cnt[j] && pos < cap)
        __stcs(reinterpret_cast<int4*>(out + pos),
               make_int4(null ? EJ_NULL_KEY : key[j], null ? EJ_NULL_KEY : p.s[j].y, p.s[j].x, p.s[j].y));
      off += (unsigned)__popc(b);
    }
    return;
  }
  static_assert(PR_ITEMS == 4, "four probes travel as vectors");
  ej_slot_emit_runs(make_int4(p.s[0].x, p.s[1].x, p.s[2].x, p.s[3].x), make_int4(p.s[0].y, p.s[1].y, p.s[2].y, p.s[3].y),
                    make_uint4(p.lo[0], p.lo[1], p.lo[2], p.lo[3]), make_uint4(p.cnt[0], p.cnt[1], p.cnt[2], p.cnt[3]),
                    make_int4(key[0], key[1], key[2], key[3]), t.rkey, off, out, cap, stage);
}

// Run descriptors of the two-pass probe: per probe one word, the key of a
// single match or the packed run {lo << 5 | min(rows, 31)} of several, and per
// 32 probes two ballots {one match, several}, so that the write pass reads no
// table for probes with one match.  Laid out as the words of whole tiles, then
// the ballots.
__device__ __forceinline__ uint2* ej_slot_ballots(void* desc, uint64_t nwtiles) {
  return reinterpret_cast<uint2*>(static_cast<uint32_t*>(desc) + nwtiles * PR_WTILE);
}

// count pass of warp tile w; DESC: also its descriptors.  Every lane returns
// the tile's rows.
template <bool OUTER, bool DESC>
__device__ __forceinline__ unsigned long long ej_slot_count(const ej_tuple* __restrict__ P, uint64_t w, uint64_t nP,
                                                            const EjSlotTable& t, void* __restrict__ desc,
                                                            uint64_t nwtiles) {
  const unsigned lane = threadIdx.x & 31u;
  EjProbeWarp p;
  int32_t key[PR_ITEMS];
  ej_slot_probe<OUTER>(P, w * PR_WTILE, nP, t, p, key);
  unsigned long long mine = 0;
#pragma unroll
  for (int j = 0; j < PR_ITEMS; j++) {
    mine += p.cnt[j];
    if (DESC) {
      const unsigned one = __ballot_sync(EJ_FULL_MASK, p.cnt[j] && p.lo[j] == INLINE_RUN);
      const unsigned run = __ballot_sync(EJ_FULL_MASK, p.cnt[j] && p.lo[j] < INLINE_RUN);
      __stcs(static_cast<unsigned int*>(desc) + w * PR_WTILE + j * 32 + lane,
             p.lo[j] < INLINE_RUN ? p.lo[j] << 5 | min(p.cnt[j], EJ_PACKED_ESCAPE) : (uint32_t)key[j]);
      if (lane == 0) ej_slot_ballots(desc, nwtiles)[w * PR_ITEMS + j] = make_uint2(one, run);
    }
  }
  return ej_warp_sum<unsigned long long>(mine);
}

// write pass of warp tile w, whose output starts at out[off], from the count
// pass's descriptors
template <bool OUTER>
__device__ __forceinline__ void ej_slot_write(const ej_tuple* __restrict__ P, const void* __restrict__ desc,
                                              uint64_t w, uint64_t nwtiles, uint64_t nP, const ej_table_view& t,
                                              unsigned long long off, ej_result* __restrict__ out, uint64_t cap,
                                              int4* stage) {
  const unsigned lane = threadIdx.x & 31u;
  const uint2* ballots = ej_slot_ballots(const_cast<void*>(desc), nwtiles) + w * PR_ITEMS;
  EjProbeWarp p;
  int32_t key[PR_ITEMS];
  bool escape = false;
#pragma unroll
  for (int j = 0; j < PR_ITEMS; j++) {
    const uint64_t idx = w * PR_WTILE + (uint64_t)j * 32 + lane;
    const bool ok = idx < nP;
    p.s[j] = ok ? __ldcs(reinterpret_cast<const int2*>(P) + idx) : make_int2(0, 0);
    const uint32_t d = __ldcs(static_cast<const unsigned int*>(desc) + idx);
    const uint2 b = __ldg(ballots + j);
    const bool one = b.x >> lane & 1u, run = b.y >> lane & 1u;
    key[j] = (int32_t)d;
    p.cnt[j] = one ? 1u : run ? d & 31u : 0u;
    p.lo[j] = one ? INLINE_RUN : d >> 5;
    escape |= run && p.cnt[j] == EJ_PACKED_ESCAPE;
    if (OUTER && ok && !one && !run) {
      p.cnt[j] = 1u;
      p.lo[j] = NULL_RUN;
    }
  }
  if (__any_sync(EJ_FULL_MASK, escape)) {  // runs of 31 rows and more: their lengths precede them
#pragma unroll
    for (int j = 0; j < PR_ITEMS; j++)
      if (p.cnt[j] == EJ_PACKED_ESCAPE) p.cnt[j] = ej_run_length(t.rkey, p.lo[j], t.run_words);
  }
  ej_slot_emit(p, key, t, off, out, cap, stage);
}
