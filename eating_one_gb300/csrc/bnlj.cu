// bnlj.cu - block nested-loop equi-join over all |R| x |S| pairs.
//
// Reference (joins/blockJoin_gpu/main_street): host tiles of PART = 2^18 per
// side (nestLoopJoin.cc:326-519); per tile a `count` kernel and a `join`
// kernel (join_gpu.cu:29-120) each stage 512 right tuples in shared memory and
// compare them with one left tuple per thread, with a presum + DtoH of the
// total in between - every compare runs twice.
//
// Here one kernel covers all pairs once, with the R block hashed (the classic
// refinement of the block nested loop: a block's tuples are found through an
// in-memory hash table instead of being compared one by one):
//   - each CTA takes one block of up to 16384 R rows and builds its table in
//     shared memory: rows grouped by bucket (top hash bits, about one row a
//     bucket) by a counting sort, with 2-byte bucket starts;
//   - S is streamed through two 16 KB shared-memory buffers filled by 1-D TMA
//     bulk copies (cp.async.bulk + mbarrier complete_tx), so the next S tile
//     lands while the current one is probed, two S tuples per thread and tile;
//   - a warp collects its matches {S key, R position} in a shared-memory
//     buffer and turns 64 to 128 of them into rows at a time, with one atomic
//     add on the cursor and coalesced stores (count-only mode sums per-thread
//     counters).  Result order is not deterministic; the result multiset is.
// Work is |S| bucket lookups per 16384 R rows instead of |S| x 16384
// compares.  2^16 x 2^20 rows over 2^16 keys, the whole call: by compares 4.81
// ms (14.4 T/s); 16 warps of four tuples a lane, one cursor atomic per 128 S
// tuples 0.112 ms (kernel 72 us); 32 warps of two, matches buffered 0.091 ms
// (kernel 51 us, 33 of them building and counting alone).  What bounds it is
// the latency of the lookups' dependent shared-memory reads at 32 warps.
// Waits on the mbarrier are bounded by the handle's wait limit and report
// EJ_ERR_TIMEOUT instead of hanging; a CTA that gave up still waits (bounded
// by EJ_DEFAULT_WAIT_LIMIT_NS) for its own copies in flight before it exits.
#include <algorithm>

#include "block_table.cuh"
#include "ej_device.cuh"
#include "ej_entry.h"

namespace {

constexpr int BN_THREADS = 1024;
constexpr int BN_WARPS = BN_THREADS / 32;
constexpr uint32_t BN_MIN_BUCKETS = 32u * BN_WARPS;
constexpr int BN_ITEMS = 2;                      // S tuples per thread and tile
constexpr int BN_STILE = BN_THREADS * BN_ITEMS;  // S tuples per shared-memory tile (16 KB)

struct BnStream {
  int4 tile[2][BN_STILE / 2];  // two S tuples per int4
  int2 buf[BN_WARPS][BT_BUF];
};
struct BnSmem {
  int32_t rval[BT_ROWS];
  int32_t rkey[BT_ROWS];
  union {
    BnStream st;
    uint32_t count[BT_ROWS];
  };
  uint16_t start[BT_ROWS + 2];
  unsigned long long bar[2];
  unsigned long long warp_tmp[BN_WARPS + 1];
  uint32_t scan_tmp[BN_WARPS];
  int timed_out;
};
static_assert(sizeof(BnSmem) <= 227 * 1024, "one CTA's shared memory");

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// non-blocking test of the phase (test_wait returns at once; try_wait may
// suspend the thread for a time of the hardware's choosing)
__device__ __forceinline__ bool mbar_test_wait(unsigned long long* bar, unsigned parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ void tma_load_1d(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// bounded wait by one thread; true when the phase completed in time (limit
// 0: only if it had completed at the first test).  The clock is read when
// the first test fails, then every 16 tests.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned long long* bar, unsigned parity,
                                                  unsigned long long limit_ns) {
  if (mbar_test_wait(bar, parity)) return true;
  if (limit_ns == 0) return false;
  const unsigned long long t0 = ej_globaltimer();
  do {
#pragma unroll 1
    for (int k = 0; k < 16; k++)
      if (mbar_test_wait(bar, parity)) return true;
  } while (ej_globaltimer() - t0 < limit_ns);
  return false;
}

template <bool USE_TMA>
__device__ __forceinline__ void issue_tile(BnSmem& sm, int buf, const ej_tuple* S, uint64_t t0, uint32_t n) {
  if (USE_TMA) {
    if (threadIdx.x == 0) {
      const uint32_t pairs = n >> 1;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_expect_tx(&sm.bar[buf], pairs * 16u);
      if (pairs) tma_load_1d(&sm.st.tile[buf][0], S + t0, pairs * 16u, &sm.bar[buf]);
      if (n & 1u) {  // odd tail tuple: plain load (TMA sizes are multiples of 16 bytes)
        const int2 last = *reinterpret_cast<const int2*>(S + t0 + n - 1);
        reinterpret_cast<int2*>(&sm.st.tile[buf][0])[n - 1] = last;
      }
    }
  } else {
    int2* dst = reinterpret_cast<int2*>(&sm.st.tile[buf][0]);
    const int2* src = reinterpret_cast<const int2*>(S + t0);
    for (uint32_t i = threadIdx.x; i < n; i += BN_THREADS) dst[i] = __ldcs(src + i);
  }
}

template <bool USE_TMA, bool COUNT_ONLY>
__global__ void __launch_bounds__(BN_THREADS, 1)
bnl_kernel(const ej_tuple* __restrict__ R, uint64_t nR, uint32_t r_block, uint32_t lg, const ej_tuple* __restrict__ S,
           uint64_t nS, uint64_t s_per_cta, ej_result* __restrict__ out, uint64_t cap, unsigned long long* cursor,
           ej_dev_status* st, unsigned long long wait_ns) {
  extern __shared__ __align__(128) unsigned char bn_smem_raw[];
  BnSmem& sm = *reinterpret_cast<BnSmem*>(bn_smem_raw);
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t rbase = (uint64_t)blockIdx.x * r_block;
  const uint64_t s_begin = (uint64_t)blockIdx.y * s_per_cta;
  const uint64_t s_end = min(nS, s_begin + s_per_cta);
  const uint64_t ntiles = s_end > s_begin ? (s_end - s_begin + BN_STILE - 1) / BN_STILE : 0;

  if (threadIdx.x == 0) {
    sm.timed_out = 0;
    if (USE_TMA) {
      mbar_init(&sm.bar[0], 1);
      mbar_init(&sm.bar[1], 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
  }
  const BtTable table = {sm.rval, sm.rkey, sm.count, sm.start, sm.scan_tmp, lg};
  const bool deep = bt_build<BN_THREADS>(table, reinterpret_cast<const int2*>(R + rbase),
                                         (uint32_t)min((uint64_t)r_block, nR - rbase));

  BtBuffer found = {sm.st.buf[threadIdx.x >> 5], 0u};
  const BtOut rows = {out, cap, cursor, nullptr};
  unsigned long long local = 0;
  if (ntiles) issue_tile<USE_TMA>(sm, 0, S, s_begin, (uint32_t)min((uint64_t)BN_STILE, s_end - s_begin));
  uint64_t t;
  for (t = 0; t < ntiles; t++) {
    const int buf = (int)(t & 1);
    const uint64_t t0 = s_begin + t * BN_STILE;
    const uint32_t n = (uint32_t)min((uint64_t)BN_STILE, s_end - t0);
    if (t + 1 < ntiles) {
      const uint64_t t1 = t0 + BN_STILE;
      issue_tile<USE_TMA>(sm, buf ^ 1, S, t1, (uint32_t)min((uint64_t)BN_STILE, s_end - t1));
    }
    if (USE_TMA) {
      if (threadIdx.x == 0 && !mbar_wait_bounded(&sm.bar[buf], (unsigned)((t >> 1) & 1u), wait_ns))
        sm.timed_out = 1;
    }
    __syncthreads();
    if (sm.timed_out) break;
    // the warp's 64 S tuples, lane l taking tuples l and 32 + l
    const uint32_t w0 = (threadIdx.x >> 5) * (32u * BN_ITEMS);
    const int2* tile = reinterpret_cast<const int2*>(sm.st.tile[buf]) + w0;
    int2 s[BN_ITEMS];
    bool ok[BN_ITEMS];
#pragma unroll
    for (int j = 0; j < BN_ITEMS; j++) {
      ok[j] = w0 + (uint32_t)j * 32u + lane < n;
      s[j] = ok[j] ? tile[j * 32 + lane] : make_int2(0, 0);
    }
    local += deep ? bt_probe<true, COUNT_ONLY, false, false>(table, s, ok, 0u, nullptr, found, rows)
                  : bt_probe<false, COUNT_ONLY, false, false>(table, s, ok, 0u, nullptr, found, rows);
    __syncthreads();  // everyone is done with `buf` before it is refilled
  }
  if (!COUNT_ONLY && found.held) bt_flush<false>(table, found, nullptr, rows);
  if (sm.timed_out && threadIdx.x == 0) {
    ej_set_status(st, EJ_ERR_TIMEOUT, 2u);
    // drain copies still in flight so none lands after the CTA exits
    for (uint64_t u = t; u < ntiles && u <= t + 1; u++)
      mbar_wait_bounded(&sm.bar[u & 1], (unsigned)((u >> 1) & 1u), EJ_DEFAULT_WAIT_LIMIT_NS);
  }
  if (COUNT_ONLY) {
    unsigned long long total;
    ej_block_exclusive_sum<BN_THREADS, unsigned long long>(local, sm.warp_tmp, &total);
    if (threadIdx.x == 0 && total) atomicAdd(cursor, total);
  }
}

template <bool USE_TMA, bool COUNT_ONLY>
ej_status launch_bnl(ej_handle* h, dim3 grid, const ej_tuple* R, uint64_t nR, uint32_t r_block, uint32_t lg,
                     const ej_tuple* S, uint64_t nS, uint64_t s_per_cta, ej_result* out, uint64_t cap, unsigned long long* cursor) {
  auto k = bnl_kernel<USE_TMA, COUNT_ONLY>;
  EJ_CUDA(h, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BnSmem)));
  k<<<grid, BN_THREADS, sizeof(BnSmem), h->stream>>>(R, nR, r_block, lg, S, nS, s_per_cta, out, cap, cursor, h->d_status,
                                                      h->wait_limit_ns);
  return ej_check_launch(h, "bnl_kernel");
}

// the nested loop over R x S; rows go to out at the positions *cursor hands
// out (not reset here, so successive calls append)
ej_status bnl_launch(ej_handle* h, const ej_tuple* R, uint64_t nR, const ej_tuple* S, uint64_t nS,
                     ej_result* out, uint64_t cap, bool count_only, unsigned long long* cursor) {
  if (nR == 0 || nS == 0) return EJ_OK;
  const uint64_t rchunks = (nR + BT_ROWS - 1) / BT_ROWS;
  if (rchunks > 0x7FFFFFFFull) return ej_fail(h, EJ_ERR_TOO_LARGE, "R too large for the nested loop");
  const uint32_t r_block = (uint32_t)((nR + rchunks - 1) / rchunks);  // blocks of even size
  const uint32_t lg = std::max(ej_ceil_log2(r_block), ej_ceil_log2(BN_MIN_BUCKETS));  // one row a bucket or less
  // one CTA per SM (its shared memory), so the S ranges are as many as fill
  // one wave; each is a whole number of tiles
  const uint64_t stiles = (nS + BN_STILE - 1) / BN_STILE;
  uint64_t splits = std::max<uint64_t>(1, (uint64_t)h->num_sms / rchunks);
  splits = std::min<uint64_t>(std::min<uint64_t>(splits, stiles), 65535);
  const uint64_t s_per_cta = ((stiles + splits - 1) / splits) * BN_STILE;
  splits = (nS + s_per_cta - 1) / s_per_cta;
  const dim3 grid((unsigned)rchunks, (unsigned)splits);
  const bool tma = ((uintptr_t)S % 16) == 0;
  if (count_only)
    return tma ? launch_bnl<true, true>(h, grid, R, nR, r_block, lg, S, nS, s_per_cta, out, cap, cursor)
               : launch_bnl<false, true>(h, grid, R, nR, r_block, lg, S, nS, s_per_cta, out, cap, cursor);
  return tma ? launch_bnl<true, false>(h, grid, R, nR, r_block, lg, S, nS, s_per_cta, out, cap, cursor)
             : launch_bnl<false, false>(h, grid, R, nR, r_block, lg, S, nS, s_per_cta, out, cap, cursor);
}

}  // namespace

static ej_status bnl_run(ej_handle* h, const ej_tuple* R, uint64_t nR, const ej_tuple* S, uint64_t nS,
                         ej_result* out, uint64_t cap, bool count_only) {
  EJ_CUDA(h, cudaMemsetAsync(h->d_words, 0, sizeof(unsigned long long), h->stream));
  // one pass: the whole nested loop is recorded as the write phase
  ej_phase_begin(h);
  for (int k = 1; k < EJ_PHASES; k++) ej_phase_mark(h, k);
  const ej_status st = bnl_launch(h, R, nR, S, nS, out, cap, count_only, h->d_words);
  ej_phase_mark(h, EJ_PHASES);
  return st;
}

ej_status ej_bnl_append(ej_handle* h, const ej_tuple* R, uint64_t nR, const ej_tuple* S, uint64_t nS,
                        ej_result* out, uint64_t cap, unsigned long long* cursor) {
  return bnl_launch(h, R, nR, S, nS, out, cap, false, cursor);
}

extern "C" ej_status ej_bnl_join(ej_handle* h, const ej_tuple* R, uint64_t nR, const ej_tuple* S, uint64_t nS,
                                 ej_result* out, uint64_t out_cap, uint64_t* out_count) {
  EJ_TRY(ej_begin(h));
  EJ_TRY(ej_check_rel(h, "R", R, nR));
  EJ_TRY(ej_check_rel(h, "S", S, nS));
  EJ_TRY(ej_check_out(h, out, out_cap, out_count));
  EJ_TRY(bnl_run(h, R, nR, S, nS, out, out_cap, false));
  uint64_t count = 0;
  EJ_TRY(ej_finish(h, &count));
  *out_count = count;
  return ej_capacity_result(h, count, out_cap);
}

extern "C" ej_status ej_bnl_join_count(ej_handle* h, const ej_tuple* R, uint64_t nR, const ej_tuple* S, uint64_t nS,
                                       uint64_t* out_count) {
  EJ_TRY(ej_begin(h));
  EJ_TRY(ej_check_rel(h, "R", R, nR));
  EJ_TRY(ej_check_rel(h, "S", S, nS));
  if (!out_count) return ej_fail(h, EJ_ERR_INVALID, "out_count is NULL");
  EJ_TRY(bnl_run(h, R, nR, S, nS, nullptr, 0, true));
  uint64_t count = 0;
  EJ_TRY(ej_finish(h, &count));
  *out_count = count;
  return EJ_OK;
}
