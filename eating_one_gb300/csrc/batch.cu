// batch.cu - many hash joins as one pipeline.
//
// The reference runs one join per process, every phase its own launch with a
// host synchronisation after it (joins/hashJoin_gpu/main_street/hj.cc:454-475).
// For a stream of joins of uneven sizes (most of them small) that is launch-
// and latency-bound.  Here a batch of joins is one fixed sequence of launches,
// whatever the number of joins in it:
//   build       every join that is not small gets a slot table (slot_table.cuh)
//               in its own part of the scratch: one launch over all joins' R
//               tiles claims the slots, two more finish keys with several rows
//               (and exit at once when no join has any)
//   probe       one launch over a task list, a task per block: whole small
//               joins (R of at most 2048 rows: table built and probed in
//               shared memory by one CTA, no radix pass) and the probe tiles
//               of the others (each warp finds its runs, reserves its rows
//               with one atomic add on its join's count and writes them, as
//               the one-pass probe of single joins does).
// Joins of more than 2^22 R rows (EJ_BATCH_MAX_ROWS) run as single joins after the
// batch's launches, on the same stream.
// Every join's rows are the rows it gives alone; their order within the join
// is not specified (warps reserve their ranges in the order they arrive).
#include <string.h>

#include <algorithm>

#include "ej_device.cuh"
#include "ej_entry.h"
#include "hash_join.cuh"
#include "slot_table.cuh"

namespace {

constexpr int BX_ITEMS = 4;                              // R rows per thread and tile (the insert: one, 4 blocks a tile)
constexpr uint32_t BX_RTILE = 256 * BX_ITEMS;            // R rows per build tile
// Larger joins run as single joins: their tables are claimed by bucket groups in
// shared memory and S is partitioned, where the batch claims slots and probes all
// over memory.  Four joins in a batch, |S| = 4 |R|, unique keys and two rows a key,
// in ms, as here, all in the batch's tables, and by radix passes as before these:
// 2^23 rows 3.14, 3.32, 4.00 and 3.36, 6.26, 4.42; 2^24 5.80, 7.90, 10.3 and 6.28, 14.0,
// 10.8; one of 2^25.5 2.05, 3.50, 3.93 and 2.81, 6.65, 3.89.  From 2^21 rows on it
// is a matter of the keys: four of 2^22 1.70 as single joins, 1.43 in the batch (radix 1.82), with two
// rows a key 1.79 and 2.70 (2.00); the served requests' keys are unique.
constexpr uint64_t BX_MAX_R = EJ_BATCH_MAX_ROWS;

// {runs' cursor of the join's table, ...}: cleared with the slots
struct BatchTableHeader {
  uint32_t cursor, pad;
};

// per join, on the device
struct BatchJoin {
  ej_table_view view;
  const ej_tuple* S;
  ej_result* out;
  unsigned long long cap;
  unsigned long long* d_count;  // the join's row cursor, then its count
  unsigned long long nS;
  unsigned long long nwtiles;  // warp tiles of the join
  unsigned long long r_row0;   // first row of the join in the marks and ranks
  const ej_tuple* R;
  unsigned long long* slot;    // the join's slots (view.pair)
  int32_t* runs;               // and their runs (view.rkey)
};

// a build tile: rows [row0, row0 + BX_RTILE) of a join's R
struct BatchTile {
  uint32_t join, row0;
};

// a task of the batch's task list: BX_TASK_TILES consecutive probe tiles of a
// join (the first of them local), or a whole small join (local = BX_SMALL_TASK)
struct BatchTask {
  uint32_t join, local;
};
// 4096 probes: a task per 1024 made the list, planned and copied up per call,
// four times as long (52000 tasks for 32 joins of 53 M probes)
constexpr uint32_t BX_TASK_TILES = 4;
constexpr uint32_t BX_SMALL_TASK = 0xFFFFFFFFu;
// joins of at most this many R rows are built and probed in shared memory
constexpr uint32_t BX_SMALL_R = 2048;

// ---- build: slot_table.cuh's steps over the tiles of all joins ---------------------

// One row a thread (as slot_insert_kernel, but over tables that L2 does not hold
// all at once): 32 served requests of 13.3 M R rows, with the clear, 420 us with
// four rows, 387 with two, 348 with one.
__global__ void __launch_bounds__(256, 8)
batch_insert_kernel(const BatchTile* __restrict__ tiles, const BatchJoin* __restrict__ joins,
                    uint32_t* __restrict__ mark, uint2* __restrict__ rank, uint32_t* __restrict__ marked) {
  const BatchTile d = tiles[blockIdx.x / BX_ITEMS];
  const BatchJoin& j = joins[d.join];
  const uint32_t i = d.row0 + blockIdx.x % BX_ITEMS * 256 + threadIdx.x;
  const bool ok[1] = {i < (uint32_t)j.view.nR};
  const int2 r = ok[0] ? __ldg(reinterpret_cast<const int2*>(j.R) + i) : make_int2(0, 0);
  const int32_t key[1] = {r.x};
  const uint32_t hv[1] = {ej_hash32((uint32_t)r.y)};
  EjSlotMark m[1];
  ej_slot_insert<1>(j.slot, j.view.npairs, key, hv, ok, m);
  if (ok[0]) mark[j.r_row0 + i] = m[0].mark;
  if (m[0].mark) rank[j.r_row0 + i] = make_uint2(m[0].rank, (uint32_t)m[0].first);
  if (__any_sync(EJ_FULL_MASK, m[0].mark != 0u) && (threadIdx.x & 31u) == 0u) *marked = 1u;
}

// the passes over the marked rows: a few blocks per SM stride over the tiles
__global__ void __launch_bounds__(256)
batch_reserve_kernel(const BatchTile* __restrict__ tiles, uint32_t ntiles, const BatchJoin* __restrict__ joins,
                     const uint32_t* __restrict__ mark, const uint2* __restrict__ rank,
                     BatchTableHeader* __restrict__ hdr, const uint32_t* __restrict__ marked) {
  if (__ldg(marked) == 0u) return;
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BatchTile d = tiles[t];
    const BatchJoin& j = joins[d.join];
    const uint32_t base = d.row0 + (threadIdx.x >> 5) * (32 * BX_ITEMS) + (threadIdx.x & 31u);
    uint32_t m[BX_ITEMS];
    uint2 r[BX_ITEMS];
#pragma unroll
    for (int q = 0; q < BX_ITEMS; q++)
      m[q] = base + 32u * q < j.view.nR ? __ldg(mark + j.r_row0 + base + 32u * q) : 0u;
#pragma unroll
    for (int q = 0; q < BX_ITEMS; q++)
      r[q] = m[q] ? __ldg(rank + j.r_row0 + base + 32u * q) : make_uint2(0u, 0u);
    ej_slot_reserve<BX_ITEMS>(reinterpret_cast<uint2*>(j.slot), m, r, j.runs, &hdr[d.join].cursor);
  }
}

__global__ void __launch_bounds__(256)
batch_place_kernel(const BatchTile* __restrict__ tiles, uint32_t ntiles, const BatchJoin* __restrict__ joins,
                   const uint32_t* __restrict__ mark, const uint2* __restrict__ rank,
                   const uint32_t* __restrict__ marked) {
  if (__ldg(marked) == 0u) return;
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const BatchTile d = tiles[t];
    const BatchJoin& j = joins[d.join];
    for (uint32_t i = d.row0 + threadIdx.x; i < min(d.row0 + BX_RTILE, (uint32_t)j.view.nR); i += 256) {
      const uint32_t m = __ldg(mark + j.r_row0 + i);
      if (m)
        j.runs[(reinterpret_cast<const uint2*>(j.slot)[m - 1u].x >> 5) +
               (__ldg(&rank[j.r_row0 + i].x) & ~EJ_SLOT_OPENER)] = j.R[i].key;
    }
  }
}

// one probe tile of a join with a slot table: each warp reserves its rows on its
// join's cursor (d_count, zeroed before the launch), so the cursor ends at the
// join's count
__device__ __forceinline__ void batch_probe_tile(const BatchJoin& j, uint32_t local, int4 (*stage)[PW_STAGE_ROWS],
                                                 ej_dev_status* st) {
  const unsigned int warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint64_t w = (uint64_t)local * PR_WARPS + warp;
  if (w >= j.nwtiles) return;
  {  // the next tile of the warp, 1 KB, lanes 0..7
    const uint64_t off = (w + PR_WARPS) * (PR_WTILE * 8) + (uint64_t)lane * 128u;
    if (lane < 8u && off < j.nS * 8) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(j.S) + off));
  }
  EjProbeWarp pw;
  int32_t key[PR_ITEMS];
  ej_slot_probe<false>(j.S, w * PR_WTILE, j.nS, ej_slots_of(j.view), pw, key);
  unsigned long long mine = 0;
#pragma unroll
  for (int q = 0; q < PR_ITEMS; q++) mine += pw.cnt[q];
  const unsigned long long total = ej_warp_sum<unsigned long long>(mine);
  if (total == 0) return;
  unsigned long long off = 0;
  if (lane == 0) {
    off = atomicAdd(j.d_count, total);
    if (off <= j.cap && off + total > j.cap) ej_set_status(st, EJ_ERR_CAPACITY, 0u);
  }
  off = __shfl_sync(EJ_FULL_MASK, off, 0);
  if (off >= j.cap) return;
  ej_slot_emit(pw, key, j.view, off, j.out, j.cap, stage[warp]);
}

// A join small enough for shared memory (nR <= BX_SMALL_R), whole, by one
// CTA: R into a chained hash table in shared memory (bucket heads and row
// links), then S probed 32 rows per warp and round: every lane walks its
// row's chain twice, first counting, then - after one atomic add on the
// join's cursor has reserved the warp's rows - writing them.  No radix pass,
// no table in global memory.
__device__ __forceinline__ void batch_small_join(const BatchJoin& j, int4* smem, ej_dev_status* st) {
  int32_t* rk = reinterpret_cast<int32_t*>(smem);
  int32_t* rv = rk + BX_SMALL_R;
  int32_t* nxt = rv + BX_SMALL_R;
  int32_t* head = nxt + BX_SMALL_R;
  const uint32_t nR = (uint32_t)j.view.nR;
  uint32_t nb = 1;
  while (nb < nR) nb <<= 1;
  for (uint32_t b = threadIdx.x; b < nb; b += PR_THREADS) head[b] = -1;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < nR; i += PR_THREADS) {
    const int2 r = reinterpret_cast<const int2*>(j.R)[i];
    rk[i] = r.x;
    rv[i] = r.y;
    nxt[i] = atomicExch(&head[ej_hash32((uint32_t)r.y) & (nb - 1)], (int)i);
  }
  __syncthreads();
  const unsigned lane = threadIdx.x & 31u;
  for (uint64_t base = (uint64_t)(threadIdx.x >> 5) * 32; base < j.nS; base += PR_THREADS) {
    const uint64_t si = base + lane;
    int2 s = make_int2(0, 0);
    uint32_t c = 0;
    int first = -1;
    if (si < j.nS) {
      s = __ldcs(reinterpret_cast<const int2*>(j.S) + si);
      first = head[ej_hash32((uint32_t)s.y) & (nb - 1)];
      for (int i = first; i >= 0; i = nxt[i]) c += rv[i] == s.y ? 1u : 0u;
    }
    const uint32_t incl = ej_warp_inclusive_sum<uint32_t>(c);
    const uint32_t total = __shfl_sync(EJ_FULL_MASK, incl, 31);
    if (total == 0) continue;
    unsigned long long off = 0;
    if (lane == 0) {
      off = atomicAdd(j.d_count, (unsigned long long)total);
      if (off <= j.cap && off + total > j.cap) ej_set_status(st, EJ_ERR_CAPACITY, 0u);
    }
    off = __shfl_sync(EJ_FULL_MASK, off, 0) + (incl - c);
    for (int i = first; c && i >= 0; i = nxt[i]) {
      if (rv[i] != s.y) continue;
      if (off < j.cap) __stcs(reinterpret_cast<int4*>(j.out + off), make_int4(rk[i], s.y, s.x, s.y));
      off++;
    }
  }
}

// The probe of a batch as one launch over a task list, one task per block,
// handed out in list order by the block scheduler: a whole small join (table
// built and probed in shared memory) or BX_TASK_TILES 1024-probe tiles of a join
// with a slot table.  The small joins come first, so that no
// large task waits behind them at the end.  (A resident grid pulling tasks
// from an atomic counter measured slower.)  32 served requests of 13.3 M
// R rows in all: four segmented radix passes, bucket bounds and this kernel over
// them 0.46 + 0.05 + 0.73 ms, slots and this kernel 0.35 + 0.55; the call 1.57 ->
// 1.19 ms.
__global__ void __launch_bounds__(PR_THREADS, 4)
batch_task_kernel(const BatchJoin* __restrict__ joins, const BatchTask* __restrict__ tasks, ej_dev_status* st) {
  __shared__ int4 smem[PR_WARPS * PW_STAGE_ROWS];  // staging rows, or a small join's table
  static_assert(4 * BX_SMALL_R * sizeof(int32_t) <= sizeof(int4) * PR_WARPS * PW_STAGE_ROWS,
                "a small join's table fits in the staging buffers");
  const BatchTask task = tasks[blockIdx.x];
  const BatchJoin& j = joins[task.join];
  if (task.local == BX_SMALL_TASK)
    batch_small_join(j, smem, st);
  else
    for (uint32_t k = 0; k < BX_TASK_TILES; k++)
      batch_probe_tile(j, task.local + k, reinterpret_cast<int4(*)[PW_STAGE_ROWS]>(smem), st);
}

}  // namespace

// Plan and launch; counts go to d_counts[i] (device).
static ej_status batch_run(ej_handle* h, const ej_join_desc* jd, uint32_t n, unsigned long long* d_counts) {
  // host-side layout of the batch
  std::vector<BatchJoin> joins(n);
  std::vector<BatchTile> tiles;
  std::vector<BatchTask> small_tasks, tile_tasks;
  std::vector<uint64_t> pair0(n), run0(n);
  std::vector<uint32_t> large;
  uint64_t nr_total = 0, pairs = 0, run_words = 0;
  for (uint32_t i = 0; i < n; i++) {
    const uint64_t nR = jd[i].nR, nS = jd[i].nS;
    BatchJoin& b = joins[i];
    b.R = jd[i].R;
    b.S = jd[i].S;
    b.nS = nS;
    b.out = jd[i].out;
    b.cap = jd[i].out_cap;
    b.d_count = d_counts + i;
    b.r_row0 = nr_total;
    b.view.kind = EJ_TABLE_HASH;
    b.view.nR = nR;
    b.nwtiles = (nS + PR_WTILE - 1) / PR_WTILE;
    pair0[i] = pairs;
    run0[i] = run_words;
    if (nR > BX_MAX_R) {
      large.push_back(i);
      continue;
    }
    if (nR && nR <= BX_SMALL_R) {  // built and probed by one CTA in shared memory
      if (nS) small_tasks.push_back({i, BX_SMALL_TASK});
      continue;
    }
    // at most half full; a bucket-bits delta above a batch's default, 1, makes it emptier
    b.view.npairs = ((uint32_t)nR << std::max(0, ej_tuned_bucket_delta(h, nR, 1) - 1)) + 1u;
    b.view.run_words = (uint32_t)ej_slot_run_words(nR);
    pairs += b.view.npairs;
    run_words += (ej_slot_run_bytes(nR) / sizeof(int32_t) + 3) & ~uint64_t(3);
    for (uint64_t r = 0; r < nR; r += BX_RTILE) tiles.push_back({i, (uint32_t)r});
    const uint32_t nptiles = (uint32_t)((nS + PR_TILE - 1) / PR_TILE);
    for (uint32_t t = 0; t < nptiles && nR; t += BX_TASK_TILES) tile_tasks.push_back({i, t});
    nr_total += nR;
  }
  if (tiles.size() > 0x7FFFFFFFull / BX_ITEMS || tile_tasks.size() + small_tasks.size() > 0x7FFFFFFFull)
    return ej_fail(h, EJ_ERR_TOO_LARGE, "batch of %llu R rows is too large", (unsigned long long)nr_total);

  // arena layout: first what one copy brings (descriptors, the task list with the
  // small joins first), then what one memset clears (headers, slots), then the rest
  const size_t ntasks = small_tasks.size() + tile_tasks.size();
  ej_plan_bytes p;
  const size_t joins_off = p.add(n * sizeof(BatchJoin));
  const size_t tiles_off = p.add(tiles.size() * sizeof(BatchTile));
  const size_t tasks_off = p.add(ntasks * sizeof(BatchTask));
  const size_t up_bytes = p.bytes;
  const size_t hdr_off = p.add(n * sizeof(BatchTableHeader));
  const size_t marked_off = p.add(sizeof(uint32_t));
  const size_t slots_off = p.add(pairs * sizeof(uint4));
  const size_t clear_bytes = p.bytes - hdr_off;
  const size_t runs_off = p.add(run_words * sizeof(int32_t));
  const size_t mark_off = p.add(nr_total * sizeof(uint32_t));
  const size_t rank_off = p.add(nr_total * sizeof(uint2));
  EJ_TRY(ej_arena_reserve(h, p.bytes));

  char* A = static_cast<char*>(h->arena);
  for (uint32_t i = 0; i < n; i++) {
    BatchJoin& b = joins[i];
    b.slot = reinterpret_cast<unsigned long long*>(A + slots_off + pair0[i] * sizeof(uint4));
    b.runs = reinterpret_cast<int32_t*>(A + runs_off) + run0[i];
    b.view.pair = reinterpret_cast<const uint4*>(b.slot);
    b.view.rkey = b.runs;
  }
  std::vector<char> up(up_bytes);
  memcpy(up.data() + joins_off, joins.data(), n * sizeof(BatchJoin));
  if (!tiles.empty()) memcpy(up.data() + tiles_off, tiles.data(), tiles.size() * sizeof(BatchTile));
  BatchTask* up_tasks = reinterpret_cast<BatchTask*>(up.data() + tasks_off);
  std::copy(tile_tasks.begin(), tile_tasks.end(), std::copy(small_tasks.begin(), small_tasks.end(), up_tasks));
  EJ_CUDA(h, cudaMemcpyAsync(A, up.data(), up_bytes, cudaMemcpyHostToDevice, h->stream));
  EJ_CUDA(h, cudaMemsetAsync(A + hdr_off, 0, clear_bytes, h->stream));
  EJ_CUDA(h, cudaMemsetAsync(d_counts, 0, n * sizeof(unsigned long long), h->stream));
  const BatchJoin* djoins = reinterpret_cast<const BatchJoin*>(A + joins_off);
  const BatchTile* dtiles = reinterpret_cast<const BatchTile*>(A + tiles_off);
  uint32_t* mark = reinterpret_cast<uint32_t*>(A + mark_off);
  uint2* rank = reinterpret_cast<uint2*>(A + rank_off);
  uint32_t* marked = reinterpret_cast<uint32_t*>(A + marked_off);
  BatchTableHeader* hdr = reinterpret_cast<BatchTableHeader*>(A + hdr_off);

  ej_phase_begin(h);
  if (!tiles.empty()) {
    const uint32_t nt = (uint32_t)tiles.size();
    const unsigned few = std::min<unsigned>(nt, (unsigned)h->num_sms * 8);
    batch_insert_kernel<<<nt * BX_ITEMS, 256, 0, h->stream>>>(dtiles, djoins, mark, rank, marked);
    EJ_TRY(ej_check_launch(h, "batch_insert_kernel"));
    batch_reserve_kernel<<<few, 256, 0, h->stream>>>(dtiles, nt, djoins, mark, rank, hdr, marked);
    EJ_TRY(ej_check_launch(h, "batch_reserve_kernel"));
    batch_place_kernel<<<few, 256, 0, h->stream>>>(dtiles, nt, djoins, mark, rank, marked);
    EJ_TRY(ej_check_launch(h, "batch_place_kernel"));
  }
  ej_phase_mark(h, 1);
  ej_phase_mark(h, 2);  // no partition pass: every table of a batch is probed in place
  ej_phase_mark(h, 3);  // one pass: recorded as the write phase
  if (ntasks) {
    batch_task_kernel<<<(unsigned)ntasks, PR_THREADS, 0, h->stream>>>(
        djoins, reinterpret_cast<const BatchTask*>(A + tasks_off), h->d_status);
    EJ_TRY(ej_check_launch(h, "batch_task_kernel"));
  }
  ej_phase_mark(h, 4);
  // the large joins take the arena over, after the launches above
  for (const uint32_t i : large)
    EJ_TRY(ej_hash_join_run(h, jd[i].R, jd[i].nR, jd[i].S, jd[i].nS, jd[i].out, jd[i].out_cap, d_counts + i, 0));
  return EJ_OK;
}

static ej_status batch_check(ej_handle* h, const ej_join_desc* joins, uint32_t n) {
  if (n && !joins) return ej_fail(h, EJ_ERR_INVALID, "joins is NULL");
  for (uint32_t i = 0; i < n; i++) {
    EJ_TRY(ej_check_rel(h, "R", joins[i].R, joins[i].nR));
    EJ_TRY(ej_check_rel(h, "S", joins[i].S, joins[i].nS));
    if (joins[i].out_cap && !joins[i].out) return ej_fail(h, EJ_ERR_INVALID, "join %u: out is NULL", i);
    if (joins[i].out && ((uintptr_t)joins[i].out % 16))
      return ej_fail(h, EJ_ERR_INVALID, "join %u: out must be 16-byte aligned", i);
  }
  return EJ_OK;
}

extern "C" ej_status ej_batch_hash_join_async(ej_handle* h, const ej_join_desc* joins, uint32_t njoins,
                                              uint64_t* d_counts) {
  EJ_TRY(ej_begin(h));
  EJ_TRY(batch_check(h, joins, njoins));
  if (njoins && !d_counts) return ej_fail(h, EJ_ERR_INVALID, "d_counts is NULL");
  if (!njoins) return EJ_OK;
  return batch_run(h, joins, njoins, reinterpret_cast<unsigned long long*>(d_counts));
}

extern "C" ej_status ej_batch_hash_join(ej_handle* h, const ej_join_desc* joins, uint32_t njoins, uint64_t* counts) {
  EJ_TRY(ej_begin(h));
  EJ_TRY(batch_check(h, joins, njoins));
  if (njoins && !counts) return ej_fail(h, EJ_ERR_INVALID, "counts is NULL");
  if (!njoins) return EJ_OK;
  // device counts live in the handle's count area: grow it when needed
  if (njoins > h->batch_counts_cap) {
    EJ_CUDA(h, cudaStreamSynchronize(h->stream));
    cudaFree(h->d_batch_counts);
    cudaFreeHost(h->h_batch_counts);
    h->d_batch_counts = nullptr;
    h->h_batch_counts = nullptr;
    h->batch_counts_cap = 0;
    EJ_CUDA(h, ej_dev_alloc(&h->d_batch_counts, njoins * sizeof(unsigned long long)));
    EJ_CUDA(h, ej_host_alloc(&h->h_batch_counts, njoins * sizeof(unsigned long long)));
    h->batch_counts_cap = njoins;
  }
  EJ_TRY(batch_run(h, joins, njoins, h->d_batch_counts));
  EJ_CUDA(h, cudaMemcpyAsync(h->h_batch_counts, h->d_batch_counts, njoins * sizeof(unsigned long long),
                             cudaMemcpyDeviceToHost, h->stream));
  EJ_TRY(ej_finish(h, nullptr));
  bool over = false;
  for (uint32_t i = 0; i < njoins; i++) {
    counts[i] = h->h_batch_counts[i];
    over |= counts[i] > joins[i].out_cap;
  }
  return over ? ej_fail(h, EJ_ERR_CAPACITY, "a join of the batch has more results than its out_cap") : EJ_OK;
}
