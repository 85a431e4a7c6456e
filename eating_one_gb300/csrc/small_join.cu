// small_join.cu - hash joins whose build side fits in shared memory (up to
// 16384 rows): one launch, no scratch.
//
// Replaces the same reference path as hash_join.cu (joins/hashJoin_gpu/
// main_street/hj.cc:171-1269) for build sides of at most BT_ROWS rows.  There
// the fixed cost is the launches: a table of 1000 rows took eleven for its
// radix passes, sort and bucket bounds, then count, scan and write, none with
// more than a few microseconds of work.  Here every CTA builds the whole
// table in its shared memory (block_table.cuh) and its warps stride over S,
// two tuples a lane, the next two loaded while these are looked up; no warp
// waits for another after the build.
// Row order is not deterministic (warps reserve their rows in the order they
// arrive), as in the one-pass probe of larger tables.  Count + rows of 1000 x
// 4001 rows 165 -> 86 us, most of what is left the two calls' launches, copies
// and synchronisations.
#include <algorithm>

#include "block_table.cuh"
#include "ej_device.cuh"
#include "small_join.cuh"

namespace {

constexpr int SJ_ITEMS = 2;  // S tuples per lane and step

// dynamic shared memory of a CTA: the columns, then the build's counters and
// the warps' buffers in the same place, then the starts and the scan's words
struct SjLayout {
  uint32_t lg, count_off, start_off, scan_off, bytes;
};

template <int THREADS>
SjLayout sj_layout(uint64_t nR) {
  constexpr uint32_t WARPS = THREADS / 32;
  SjLayout l;
  l.lg = std::max(ej_ceil_log2(nR), ej_ceil_log2(std::max(BT_MIN_BUCKETS, 32u * WARPS)));
  const uint32_t n16 = ((uint32_t)nR + 3u) & ~3u;
  l.count_off = n16 * 8u;
  const uint32_t mid = std::max<uint32_t>(4u << l.lg, WARPS * BT_BUF * sizeof(int2));
  l.start_off = l.count_off + mid;
  l.scan_off = l.start_off + ((2u << l.lg) + 16u);
  l.bytes = l.scan_off + WARPS * 4u;
  return l;
}

// the CTA's share of S; returns the lane's matches (COUNT_ONLY)
template <int THREADS, bool DEEP, bool COUNT_ONLY, bool OUTER>
__device__ __forceinline__ unsigned long long sj_scan(const BtTable& t, const int2* __restrict__ S, uint32_t nS,
                                                      BtBuffer& found, const BtOut& out) {
  const uint32_t lane = threadIdx.x & 31u;
  constexpr uint32_t STEP = 32 * SJ_ITEMS;  // tuples per warp and step
  const uint64_t stride = (uint64_t)gridDim.x * (THREADS / 32) * STEP;
  uint64_t base = ((uint64_t)blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5)) * STEP;
  unsigned long long local = 0;
  int2 s[SJ_ITEMS];
  bool ok[SJ_ITEMS];
#pragma unroll
  for (int j = 0; j < SJ_ITEMS; j++) {
    const uint64_t i = base + 32u * j + lane;
    ok[j] = i < nS;
    s[j] = ok[j] ? __ldg(S + i) : make_int2(0, 0);
  }
  while (base < nS) {
    int2 sn[SJ_ITEMS];
    bool okn[SJ_ITEMS];
#pragma unroll
    for (int j = 0; j < SJ_ITEMS; j++) {
      const uint64_t i = base + stride + 32u * j + lane;
      okn[j] = i < nS;
      sn[j] = okn[j] ? __ldg(S + i) : make_int2(0, 0);
    }
    local += bt_probe<DEEP, COUNT_ONLY, OUTER, true>(t, s, ok, (uint32_t)base, S, found, out);
#pragma unroll
    for (int j = 0; j < SJ_ITEMS; j++) {
      s[j] = sn[j];
      ok[j] = okn[j];
    }
    base += stride;
  }
  return local;
}

// (48 registers, 40 for the count, so that 256-thread CTAs fill 40 or 48 warps an SM:
// 1000 rows and 2^28 S tuples, a tenth of them matching, 1.59 ms instead of 1.71)
template <int THREADS, bool COUNT_ONLY, bool OUTER>
__global__ void __launch_bounds__(THREADS, THREADS == 1024 ? 1 : COUNT_ONLY ? 6 : 5)
small_join_kernel(const int2* __restrict__ R, uint32_t nR, const int2* __restrict__ S, uint32_t nS, SjLayout l,
                  BtOut out) {
  extern __shared__ __align__(16) unsigned char sj_smem[];
  __shared__ unsigned long long warp_tmp[THREADS / 32 + 1];
  const uint32_t n16 = (nR + 3u) & ~3u;
  int32_t* rval = reinterpret_cast<int32_t*>(sj_smem);
  const BtTable t = {rval, rval + n16, reinterpret_cast<uint32_t*>(sj_smem + l.count_off),
                     reinterpret_cast<uint16_t*>(sj_smem + l.start_off),
                     reinterpret_cast<uint32_t*>(sj_smem + l.scan_off), l.lg};
  const bool deep = bt_build<THREADS>(t, R, nR);
  BtBuffer found = {reinterpret_cast<int2*>(sj_smem + l.count_off) + (threadIdx.x >> 5) * BT_BUF, 0u};
  const unsigned long long local = deep ? sj_scan<THREADS, true, COUNT_ONLY, OUTER>(t, S, nS, found, out)
                                        : sj_scan<THREADS, false, COUNT_ONLY, OUTER>(t, S, nS, found, out);
  if (COUNT_ONLY) {
    unsigned long long total;
    ej_block_exclusive_sum<THREADS, unsigned long long>(local, warp_tmp, &total);
    if (threadIdx.x == 0 && total) atomicAdd(out.cursor, total);
  } else if (found.held) {
    bt_flush<true>(t, found, S, out);
  }
}

// most rows of the 256-thread CTAs (see sj_run)
constexpr uint64_t SJ_SHORT_ROWS = 4096;

template <int THREADS, bool COUNT_ONLY, bool OUTER>
ej_status sj_launch(ej_handle* h, const ej_tuple* R, uint64_t nR, const ej_tuple* S, uint64_t nS, const BtOut& out) {
  const SjLayout l = sj_layout<THREADS>(nR);
  auto k = small_join_kernel<THREADS, COUNT_ONLY, OUTER>;
  // the attribute is the function's, for every handle and thread: always its most
  const SjLayout most = sj_layout<THREADS>(THREADS == 256 ? SJ_SHORT_ROWS : BT_ROWS);
  EJ_CUDA(h, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most.bytes));
  // as many CTAs as are resident at once (1 KB of each SM's 228 KB is taken
  // per CTA by the system), fewer when S is short
  const uint64_t per_sm = std::max<uint64_t>(1, std::min<uint64_t>(2048 / THREADS, (227u * 1024u) / (l.bytes + 1280u)));
  const uint64_t want = (nS + (uint64_t)THREADS * SJ_ITEMS - 1) / ((uint64_t)THREADS * SJ_ITEMS);
  const unsigned blocks = (unsigned)std::min<uint64_t>(want, per_sm * h->num_sms);
  k<<<blocks, THREADS, l.bytes, h->stream>>>(reinterpret_cast<const int2*>(R), (uint32_t)nR,
                                             reinterpret_cast<const int2*>(S), (uint32_t)nS, l, out);
  return ej_check_launch(h, "small_join_kernel");
}

template <bool COUNT_ONLY, bool OUTER>
ej_status sj_run(ej_handle* h, const ej_tuple* R, uint64_t nR, const ej_tuple* S, uint64_t nS, const BtOut& out) {
  // tables up to 4096 rows (56 KB) leave room for three or more CTAs of 256
  // threads, whose build barriers are cheaper and which spread a short S over
  // more SMs
  return nR <= SJ_SHORT_ROWS ? sj_launch<256, COUNT_ONLY, OUTER>(h, R, nR, S, nS, out)
                             : sj_launch<1024, COUNT_ONLY, OUTER>(h, R, nR, S, nS, out);
}

}  // namespace

bool ej_small_join_applies(const ej_handle* h, uint64_t nR) {
  return nR <= BT_ROWS && h->opt_partition_bits < 0 && !h->opt_bucket_delta_set && h->opt_build == 0 &&
         h->opt_table == 0 && h->opt_probe_warps == 0;
}

ej_status ej_small_join(ej_handle* h, const ej_tuple* R, uint64_t nR, const ej_tuple* S, uint64_t nS, bool outer,
                        bool count_only, ej_result* out, uint64_t cap, unsigned long long* cursor) {
  EJ_CUDA(h, cudaMemsetAsync(cursor, 0, sizeof(unsigned long long), h->stream));
  // one pass: recorded as the count phase or the write phase
  ej_phase_begin(h);
  for (int k = 1; k < EJ_PHASES - (count_only ? 1 : 0); k++) ej_phase_mark(h, k);
  const BtOut o = {out, cap, cursor, count_only ? nullptr : h->d_status};
  if (nS && (nR || outer)) {
    if (count_only)
      EJ_TRY(sj_run<true, false>(h, R, nR, S, nS, o));
    else
      EJ_TRY(outer ? sj_run<false, true>(h, R, nR, S, nS, o) : sj_run<false, false>(h, R, nR, S, nS, o));
  }
  for (int k = EJ_PHASES - (count_only ? 1 : 0); k <= EJ_PHASES; k++) ej_phase_mark(h, k);
  return EJ_OK;
}
