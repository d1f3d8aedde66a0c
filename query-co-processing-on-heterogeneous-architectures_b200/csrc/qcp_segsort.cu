// Per-query sort of the output ids.
//
// The reference returns hit counts only; this library returns every query's
// hits as ascending input ids.  The traversal writes each query's ids in
// arbitrary order into its CSR slice; this file sorts every slice in place.
// The ids of one slice are distinct and lie in [0, n), so only the low
// `idbits` = ceil(log2 n) bits carry order.
//
//   slice <= kTinyCap ids   one warp bucket-sorts it in shared memory (256
//                           buckets over the slice's own id range, a few ids
//                           each, insertion-sorted);
//   slice <= kSmallCap ids  one CTA bucket-sorts it the same way (2048
//                           buckets).  In both, a slice whose ids crowd into
//                           few buckets is radix-sorted instead.
//   larger slices           1. window partition: ids are split by
//                              id >> wbits (wbits = min(idbits, 18)) into
//                              G = 2^(idbits - wbits) windows: tile
//                              histograms -> per-slice window bases -> every
//                              tile regrouped by window in shared memory and
//                              written as contiguous runs into the scratch
//                              buffer;
//                           2. each (slice, window) of more than
//                              kWinWarpMax ids is sorted through a bitmap of
//                              its 2^wbits possible ids: every id sets its
//                              bit, every thread counts the set bits of its
//                              words, and after a CTA prefix enumerates them
//                              in order -- no comparisons; the smaller
//                              windows are bucket-sorted by one warp each.
#include "qcp_internal.cuh"
#include "qcp_tree.cuh"

namespace qcp {

namespace {

// ---- tiny slices (one warp each) --------------------------------------------
constexpr uint32_t kTinyCap = 1024;                    // ids of a slice sorted by one warp
constexpr uint32_t kTinyBuckets = 256;                 // buckets of the warp's counting pass
constexpr uint32_t kTinyWarps = 8;                     // warps per CTA
constexpr uint32_t kWinWarpMax = 512;                  // windows of at most this many ids: one warp each
// ---- small slices ----------------------------------------------------------
constexpr uint32_t kSmallCap = kSmallSliceCap;
constexpr uint32_t kSmallThreads = 256;
constexpr uint32_t kSmallWarps = kSmallThreads / 32;
constexpr uint32_t kBucketBits = 11;
constexpr uint32_t kBuckets = 1u << kBucketBits;
// ---- window partition ------------------------------------------------------
constexpr uint32_t kWinBits = 18;
// 128 threads x 16 ids per tile, 10 CTAs per SM: the partition's per-tile
// chain (counts, scan, one global atomic per window, barriers) is latency-
// bound, and more, smaller CTAs keep more chains in flight per SM
constexpr uint32_t kTile = kSortTile;
constexpr uint32_t kTileThreads = 128;
constexpr uint32_t kTileBlocks = 10;  // launch bound of k_win_scatter (registers for 10 CTAs per SM)
constexpr uint32_t kTileWarps = kTileThreads / 32;
constexpr uint32_t kPerWarpMaxG = 256;  // per-warp window counters up to this G
// ---- window sort ------------------------------------------------------------
// One instantiation per window size 2^BITS ids (BITS = 16, 17, 18).  Each
// thread owns kLaneWords bitmap words (32 for 2^17- and 2^18-id windows, 16
// for 2^16): a window's per-window bookkeeping is paid per warp, so fewer
// warps per window cost fewer instructions per id, and more bits per thread
// even out the enumeration's lanes.  Shared memory sets the resident CTAs per
// SM (kBlocks: 3, 6, 10); the launch takes the occupancy API's count.
template <uint32_t BITS>
struct WinCfg {
  static constexpr uint32_t kWords = (1u << BITS) / 32;            // bitmap words
  static constexpr uint32_t kLaneWords = BITS >= 17 ? 32u : 16u;   // bitmap words per thread
  static constexpr uint32_t kThreads = kWords / kLaneWords;        // 256, 128, 128
  static constexpr uint32_t kWarps = kThreads / 32;
  static constexpr uint32_t kBlocks = BITS >= 18 ? 3u : (BITS == 17 ? 6u : 10u);  // resident CTAs per SM
  // the launch bound: registers for kBlocks CTAs per SM (shared memory allows
  // no more); tighter caps (~40 registers) measured 5 % slower
  static constexpr uint32_t kStage = BITS >= 18 ? 6144u : (BITS == 17 ? 3072u : 1408u);  // staged output ids
  static constexpr uint32_t kPrefetch = 4096u >> (18 - BITS);      // ids of the next window loaded ahead
};
constexpr uint32_t kBatch = 8;                         // ids per thread per load round
constexpr uint32_t kNone = 0xffffffffu;                // empty register slot

using Job = SortJob;

// ============================================================================
// Small slices: bucket sort
// ============================================================================
// Ids are often not spread over [0, n): objects loaded region by region give
// a box a few short id ranges.  Buckets over all of [0, n) then hold hundreds
// of ids each and their insertion sorts dominate (5,000 boxes over 2,000,003
// points in 64 id-contiguous clusters: k_sort_small 21.5 ms, k_sort_tiny 2.7
// ms, k_win_sort_warp 1.3 ms).  So a slice with a bucket of more than
// kCrowded ids is counted again into buckets over its own range [min, max],
// and one that is crowded all the same (several ranges far apart) takes
// stable 8-bit radix passes over the bits of max - min.  kCrowded: a bucket
// of 32 ids costs its lane about 256 insertion steps, what three radix passes
// cost the warp.  The batch above: 29.3 -> 2.9 ms (0.18, 0.10 and 0.05 ms in
// the three kernels).
constexpr uint32_t kCrowded = 32;
struct BucketSmem {
  uint32_t stage[kSmallCap];
  uint32_t cnt[kBuckets];   // bucket counts, then next slots; radix: [warp][digit]
  uint32_t red[3 * kSmallWarps];
};

// Slices of at most kTinyCap ids, one warp each (no CTA barriers): the ids
// are loaded into registers (32 per lane, all loads in flight together) and
// counted into kTinyBuckets buckets, a warp scan gives the bucket bases,
// every id takes the next slot of its bucket, each lane insertion-sorts its 8
// buckets (a few ids each) and the slice leaves in coalesced stores.  Jobs of
// more ids are k_sort_small's.
// CTAs per SM (registers and shared memory): 4 for slices (3 cost their sort
// a second wave: 356 -> 540 us on 100,000 slices of 640 ids), 6 for windows.
constexpr uint32_t kTinyBlocks = 4;
constexpr uint32_t kWinWarpBlocks = 6;
template <uint32_t CAP>
struct TinySmem {
  uint32_t stage[kTinyWarps][CAP];
  uint32_t cnt[kTinyWarps][kTinyBuckets];
  uint32_t base[kTinyWarps][kTinyBuckets];
};

// Bits needed for values 0..range.
__device__ __forceinline__ uint32_t bits_of(uint32_t range) { return 32u - (uint32_t)__clz((int)range); }

// Position mask of the active lanes that hold the same 8-bit digit as this
// one (one ballot per bit).
__device__ __forceinline__ uint32_t digit_peers(uint32_t active, uint32_t d) {
  uint32_t peers = active;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const uint32_t bit = (d >> b) & 1u;
    const uint32_t bal = __ballot_sync(active, bit);
    peers &= bit ? bal : ~bal;
  }
  return peers;
}

// Stable placement of this warp's ids (v[k] at position 32 k + lane of the
// warp's run, kNone past its end) by their digit: next[d] is the next free
// slot of digit d and advances in position order.
template <uint32_t K>
__device__ __forceinline__ void place_by_digit(const uint32_t (&v)[K], uint32_t lo, uint32_t shift, uint32_t* next,
                                               uint32_t* stage, uint32_t lane) {
  const uint32_t lt = lane_lt_mask();
#pragma unroll
  for (uint32_t k = 0; k < K; ++k) {
    const bool valid = v[k] != kNone;
    const uint32_t active = __ballot_sync(0xffffffffu, valid);
    if (valid) {
      const uint32_t d = ((v[k] - lo) >> shift) & 255u;
      const uint32_t peers = digit_peers(active, d);
      const uint32_t at = next[d] + __popc(peers & lt);
      __syncwarp(active);
      if (lane == (uint32_t)(__ffs(peers) - 1)) next[d] = at + __popc(peers);
      stage[at] = v[k];
      __syncwarp(active);
    }
  }
}

// Lowest and highest id of v over the warp (kNone: empty, the least as a
// signed value).
template <uint32_t K>
__device__ __forceinline__ void warp_range(const uint32_t (&v)[K], uint32_t* lo, uint32_t* hi) {
  uint32_t a = kNone;
  int32_t b = -1;
#pragma unroll
  for (uint32_t k = 0; k < K; ++k) {
    a = min(a, v[k]);
    b = max(b, (int32_t)v[k]);
  }
  *lo = __reduce_min_sync(0xffffffffu, a);
  *hi = (uint32_t)__reduce_max_sync(0xffffffffu, b);
}

// The warp's ids into registers, all loads in flight at once (position 32 k
// + lane in v[k]).
template <uint32_t K>
__device__ __forceinline__ void load_slice(uint32_t (&v)[K], const int32_t* src, uint32_t size, uint32_t lane) {
#pragma unroll
  for (uint32_t k = 0; k < K; ++k) {
    const uint32_t i = lane + 32 * k;
    v[k] = (i < size) ? (uint32_t)__ldg(src + i) : kNone;
  }
}

// Buckets of (id - lo) >> bshift: c[] = the counts of this lane's buckets,
// *most = the largest of all.  The counters are zero on entry and on return.
template <uint32_t K>
__device__ __forceinline__ void count_buckets(const uint32_t (&v)[K], uint32_t lo, uint32_t bshift, uint32_t* cnt,
                                              uint32_t (&c)[kTinyBuckets / 32], uint32_t* most, uint32_t lane) {
  constexpr uint32_t kPer = kTinyBuckets / 32;
#pragma unroll
  for (uint32_t k = 0; k < K; ++k)
    if (v[k] != kNone) atomicAdd(&cnt[(v[k] - lo) >> bshift], 1u);
  __syncwarp();
  uint32_t m = 0;
#pragma unroll
  for (uint32_t k = 0; k < kPer; ++k) {
    c[k] = cnt[lane * kPer + k];
    m = max(m, c[k]);
    cnt[lane * kPer + k] = 0;
  }
  *most = __reduce_max_sync(0xffffffffu, m);
}

// The counted slice into stage, in order: bucket bases, every id to the next
// slot of its bucket, an insertion sort of each lane's buckets.
template <uint32_t K>
__device__ __forceinline__ void sort_buckets(const uint32_t (&v)[K], uint32_t lo, uint32_t bshift,
                                             const uint32_t (&c)[kTinyBuckets / 32], uint32_t* stage, uint32_t* base,
                                             uint32_t lane) {
  constexpr uint32_t kPer = kTinyBuckets / 32;
  uint32_t t = 0;
#pragma unroll
  for (uint32_t k = 0; k < kPer; ++k) t += c[k];
  uint32_t tot;
  uint32_t run = warp_excl_sum(t, &tot);
#pragma unroll
  for (uint32_t k = 0; k < kPer; ++k) {
    base[lane * kPer + k] = run;
    run += c[k];
  }
  __syncwarp();
#pragma unroll
  for (uint32_t k = 0; k < K; ++k)
    if (v[k] != kNone) stage[atomicAdd(&base[(v[k] - lo) >> bshift], 1u)] = v[k];
  __syncwarp();
#pragma unroll
  for (uint32_t k = 0; k < kPer; ++k) {
    const uint32_t n = c[k];
    const uint32_t b0 = base[lane * kPer + k] - n;
    for (uint32_t i = 1; i < n; ++i) {
      const uint32_t key = stage[b0 + i];
      uint32_t jj = i;
      while (jj > 0 && stage[b0 + jj - 1] > key) {
        stage[b0 + jj] = stage[b0 + jj - 1];
        --jj;
      }
      stage[b0 + jj] = key;
    }
  }
  __syncwarp();
}

// A slice whose buckets are crowded, into stage: buckets over its own range,
// or radix passes (least significant digit first) where those are crowded
// too.  Kept out of line so that the spread slices' code stays within the
// registers of kTinyBlocks CTAs per SM.
template <uint32_t CAP>
__device__ __noinline__ void warp_sort_crowded(const int32_t* src, uint32_t size, uint32_t* stage, uint32_t* cnt,
                                               uint32_t* base, uint32_t lane) {
  constexpr uint32_t kPer = kTinyBuckets / 32;
  constexpr uint32_t kPerLane = CAP / 32;
  uint32_t v[kPerLane], c[kPer];
  uint32_t lo, hi, most;
  load_slice(v, src, size, lane);
  warp_range(v, &lo, &hi);
  const uint32_t rbits = bits_of(hi - lo);
  const uint32_t bshift = rbits > 8 ? rbits - 8 : 0;
  __syncwarp();
  count_buckets(v, lo, bshift, cnt, c, &most, lane);
  if (most <= kCrowded) {
    sort_buckets(v, lo, bshift, c, stage, base, lane);
    return;
  }
  for (uint32_t shift = 0; shift < rbits; shift += 8) {  // warp-uniform
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k) base[lane * kPer + k] = 0;
    __syncwarp();
#pragma unroll
    for (uint32_t k = 0; k < kPerLane; ++k)
      if (v[k] != kNone) atomicAdd(&base[((v[k] - lo) >> shift) & 255u], 1u);
    __syncwarp();
    uint32_t t = 0;
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k) t += base[lane * kPer + k];
    uint32_t tot;
    uint32_t run = warp_excl_sum(t, &tot);
#pragma unroll
    for (uint32_t k = 0; k < kPer; ++k) {
      const uint32_t b = base[lane * kPer + k];
      base[lane * kPer + k] = run;
      run += b;
    }
    __syncwarp();
    place_by_digit<kPerLane>(v, lo, shift, base, stage, lane);
    __syncwarp();
#pragma unroll
    for (uint32_t k = 0; k < kPerLane; ++k)
      if (lane + 32 * k < size) v[k] = stage[lane + 32 * k];
    __syncwarp();
  }
}

// One warp sorts the size <= CAP (<= kTinyCap) distinct ids at src into dst
// (src may equal dst), as described above; bucket of id: (id - lo) >>
// bshift.  The warp's counters are zero on entry and on return.
template <uint32_t CAP>
__device__ __forceinline__ void warp_bucket_sort(const int32_t* src, int32_t* dst, uint32_t size, uint32_t lo,
                                                 uint32_t bshift, uint32_t* stage, uint32_t* cnt, uint32_t* base,
                                                 uint32_t lane) {
  static_assert(CAP % 32 == 0 && CAP <= kTinyCap, "one warp's stage holds kTinyCap ids");
  uint32_t v[CAP / 32], c[kTinyBuckets / 32];
  uint32_t most;
  load_slice(v, src, size, lane);
  count_buckets(v, lo, bshift, cnt, c, &most, lane);
  if (most <= kCrowded) sort_buckets(v, lo, bshift, c, stage, base, lane);
  else warp_sort_crowded<CAP>(src, size, stage, cnt, base, lane);
  for (uint32_t i = lane; i < size; i += 32) __stcs(dst + i, (int32_t)stage[i]);
  __syncwarp();
}

__global__ void __launch_bounds__(kTinyWarps * 32, kTinyBlocks) k_sort_tiny(const Job* __restrict__ jobs,
                                                               const uint32_t* __restrict__ njobs_p,
                                                               int32_t* out, uint32_t idbits) {
  const uint32_t njobs = *njobs_p;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& sm = *reinterpret_cast<TinySmem<kTinyCap>*>(smem_raw);
  const uint32_t lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  constexpr uint32_t kPer = kTinyBuckets / 32;
  const uint32_t bshift = idbits > 8 ? idbits - 8 : 0;
#pragma unroll
  for (uint32_t k = 0; k < kPer; ++k) sm.cnt[wp][lane * kPer + k] = 0;
  __syncwarp();
  const uint32_t warps = gridDim.x * kTinyWarps;
  for (uint32_t j = blockIdx.x * kTinyWarps + wp; j < njobs; j += warps) {
    const Job jb = jobs[j];
    if (jb.size > kTinyCap) continue;  // warp-uniform
    warp_bucket_sort<kTinyCap>(out + jb.off, out + jb.off, jb.size, 0u, bshift, sm.stage[wp], sm.cnt[wp], sm.base[wp],
                               lane);
  }
}

// Programmatic dependent launch: the next kernel of the stream may start once
// every CTA of this one has said so or ended; and the wait for everything
// before it.
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_prerequisites() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Windows of at most kWinWarpMax ids (listed by k_win_split), one warp
// each: the window's ids at src + wbase[g] in ascending order to
// dst + wbase[g].  It may run beside k_win_sort, launched before it, once that
// one's CTAs are all on the SMs; what it reads is complete before k_win_sort
// starts, and it ends after k_win_sort, so what follows waits for both.
__global__ void __launch_bounds__(kTinyWarps * 32, kWinWarpBlocks) k_win_sort_warp(const uint32_t* __restrict__ list,
                                                                   const uint32_t* __restrict__ nlist_p, uint32_t G,
                                                                   uint32_t wbits, const uint32_t* __restrict__ whist,
                                                                   const unsigned long long* __restrict__ wbase,
                                                                   const int32_t* __restrict__ src, int32_t* dst) {
  const uint32_t nlist = *nlist_p;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  auto& sm = *reinterpret_cast<TinySmem<kWinWarpMax>*>(smem_raw);
  const uint32_t lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  constexpr uint32_t kPer = kTinyBuckets / 32;
  const uint32_t bshift = wbits > 8 ? wbits - 8 : 0;
#pragma unroll
  for (uint32_t k = 0; k < kPer; ++k) sm.cnt[wp][lane * kPer + k] = 0;
  __syncwarp();
  const uint32_t warps = gridDim.x * kTinyWarps;
  for (uint32_t i = blockIdx.x * kTinyWarps + wp; i < nlist; i += warps) {
    const uint32_t g = list[i];
    const unsigned long long off = wbase[g];
    const uint32_t lo = (g & (G - 1)) << wbits;
    warp_bucket_sort<kWinWarpMax>(src + off, dst + off, whist[g], lo, bshift, sm.stage[wp], sm.cnt[wp], sm.base[wp],
                                  lane);
  }
  wait_for_prerequisites();
}

// The (job, window) pairs into two lists: windows of 1..kWinWarpMax ids for
// k_win_sort_warp, larger ones for k_win_sort (one atomic per warp and
// list).  With big_ids, the ids of the large windows are added to it.
__global__ void k_win_split(const uint32_t* __restrict__ njobs_p, uint32_t G, const uint32_t* __restrict__ whist,
                            uint32_t* big, uint32_t* nbig, uint32_t* small, uint32_t* nsmall,
                            unsigned long long* big_ids) {
  const uint32_t total = *njobs_p * G;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t g0 = blockIdx.x * blockDim.x; g0 < total; g0 += stride) {  // warp-uniform rounds
    const uint32_t g = g0 + threadIdx.x;
    const uint32_t sz = g < total ? whist[g] : 0u;
    const bool is_small = sz >= 1 && sz <= kWinWarpMax, is_big = sz > kWinWarpMax;
    const uint32_t ms = __ballot_sync(0xffffffffu, is_small), mb = __ballot_sync(0xffffffffu, is_big);
    uint32_t bs = 0, bb = 0;
    if (lane == 0) {
      if (ms) bs = atomicAdd(nsmall, (uint32_t)__popc(ms));
      if (mb) bb = atomicAdd(nbig, (uint32_t)__popc(mb));
    }
    bs = __shfl_sync(0xffffffffu, bs, 0);
    bb = __shfl_sync(0xffffffffu, bb, 0);
    const uint32_t lt = lane_lt_mask();
    if (is_small) small[bs + __popc(ms & lt)] = g;
    if (is_big) big[bb + __popc(mb & lt)] = g;
    if (big_ids) {
      const uint32_t ids = __reduce_add_sync(0xffffffffu, is_big ? sz : 0u);
      if (lane == 0 && ids) atomicAdd(big_ids, (unsigned long long)ids);
    }
  }
}

// One CTA per slice of kTinyCap < size <= kSmallCap ids: as warp_bucket_sort,
// with the CTA's kSmallWarps warps and kBuckets buckets.  The ids stay in
// registers (warp w holds positions [w * kWarpRun, (w + 1) * kWarpRun) of
// the slice), so every slice is read once.  jobs_end: one past the last job;
// job j is jobs_end[-1 - j].
constexpr uint32_t kWarpRun = kSmallCap / kSmallWarps;
__global__ void __launch_bounds__(kSmallThreads, 4) k_sort_small(const Job* __restrict__ jobs_end,
                                                                 const uint32_t* __restrict__ njobs_p,
                                                                 int32_t* out, uint32_t idbits) {
  const uint32_t njobs = *njobs_p;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BucketSmem& s = *reinterpret_cast<BucketSmem*>(smem_raw);
  const uint32_t tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  constexpr uint32_t kPer = kBuckets / kSmallThreads;  // buckets per thread
  constexpr uint32_t kPerLane = kWarpRun / 32;
  static_assert(kBuckets == kSmallWarps * 256, "the radix counters reuse the bucket counters");
  // exclusive sum of one value per thread over the CTA (red[0..kSmallWarps))
  auto excl_sum = [&](uint32_t t) -> uint32_t {
    uint32_t wtot;
    const uint32_t ex = warp_excl_sum(t, &wtot);
    if (lane == 0) s.red[wp] = wtot;
    __syncthreads();
    uint32_t run = ex;
    for (uint32_t k = 0; k < wp; ++k) run += s.red[k];
    return run;
  };
  for (uint32_t j = blockIdx.x; j < njobs; j += gridDim.x) {
    const Job jb = jobs_end[-1 - (long long)j];
    const uint32_t size = jb.size;
    int32_t* slice = out + jb.off;
    // 1. the slice into registers, bucket counts
    uint32_t v[kPerLane];
#pragma unroll
    for (uint32_t k = 0; k < kPerLane; ++k) {
      const uint32_t i = wp * kWarpRun + k * 32 + lane;
      v[k] = (i < size) ? (uint32_t)slice[i] : kNone;
    }
    uint32_t c[kPer];  // each thread owns kPer consecutive buckets
    uint32_t lo = 0, rbits = idbits;
    uint32_t t, bshift;
    auto count = [&]() -> bool {
      bshift = rbits > kBucketBits ? rbits - kBucketBits : 0;
#pragma unroll
      for (uint32_t k = 0; k < kPer; ++k) s.cnt[k * kSmallThreads + tid] = 0;
      __syncthreads();
#pragma unroll
      for (uint32_t k = 0; k < kPerLane; ++k)
        if (v[k] != kNone) atomicAdd(&s.cnt[(v[k] - lo) >> bshift], 1u);
      __syncthreads();
      uint32_t most = 0;
      t = 0;
#pragma unroll
      for (uint32_t k = 0; k < kPer; ++k) {
        c[k] = s.cnt[tid * kPer + k];
        t += c[k];
        most = max(most, c[k]);
      }
      return __syncthreads_or(most > kCrowded);
    };
    bool crowded = count();
    if (crowded) {
      uint32_t hi;
      warp_range(v, &lo, &hi);
      if (lane == 0) {
        s.red[kSmallWarps + wp] = lo;
        s.red[2 * kSmallWarps + wp] = hi;
      }
      __syncthreads();
      // (a warp without ids: lo = hi = kNone)
#pragma unroll
      for (uint32_t k = 0; k < kSmallWarps; ++k) {
        lo = min(lo, s.red[kSmallWarps + k]);
        hi = (uint32_t)max((int32_t)hi, (int32_t)s.red[2 * kSmallWarps + k]);
      }
      rbits = bits_of(hi - lo);
      crowded = count();
    }
    // 2. bucket bases
    if (!crowded) {
      uint32_t run = excl_sum(t);
#pragma unroll
      for (uint32_t k = 0; k < kPer; ++k) {
        s.cnt[tid * kPer + k] = run;
        run += c[k];
      }
      __syncthreads();
      // 3. every id to the next slot of its bucket
#pragma unroll
      for (uint32_t k = 0; k < kPerLane; ++k)
        if (v[k] != kNone) s.stage[atomicAdd(&s.cnt[(v[k] - lo) >> bshift], 1u)] = v[k];
      __syncthreads();
      // 4. insertion sort of each bucket [slot - count, slot)
#pragma unroll
      for (uint32_t k = 0; k < kPer; ++k) {
        const uint32_t n = c[k];
        const uint32_t b0 = s.cnt[tid * kPer + k] - n;
        for (uint32_t i = 1; i < n; ++i) {
          const uint32_t key = s.stage[b0 + i];
          uint32_t jj = i;
          while (jj > 0 && s.stage[b0 + jj - 1] > key) {
            s.stage[b0 + jj] = s.stage[b0 + jj - 1];
            --jj;
          }
          s.stage[b0 + jj] = key;
        }
      }
      __syncthreads();
    } else {
      // crowded: radix passes, least significant digit first; counters per
      // (warp, digit), slots in (digit, warp) order
      for (uint32_t shift = 0; shift < rbits; shift += 8) {  // CTA-uniform
        uint32_t* next = s.cnt + wp * 256;
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) s.cnt[k * kSmallThreads + tid] = 0;
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kPerLane; ++k)
          if (v[k] != kNone) atomicAdd(&next[((v[k] - lo) >> shift) & 255u], 1u);
        __syncthreads();
        t = 0;
#pragma unroll
        for (uint32_t w = 0; w < kSmallWarps; ++w) t += s.cnt[w * 256 + tid];
        uint32_t run = excl_sum(t);
#pragma unroll
        for (uint32_t w = 0; w < kSmallWarps; ++w) {
          const uint32_t n = s.cnt[w * 256 + tid];
          s.cnt[w * 256 + tid] = run;
          run += n;
        }
        __syncthreads();
        place_by_digit<kPerLane>(v, lo, shift, next, s.stage, lane);
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kPerLane; ++k) {
          const uint32_t i = wp * kWarpRun + k * 32 + lane;
          if (i < size) v[k] = s.stage[i];
        }
        __syncthreads();
      }
    }
    for (uint32_t i = tid; i < size; i += kSmallThreads) __stcs(slice + i, (int32_t)s.stage[i]);
    __syncthreads();
  }
}

// ============================================================================
// Window partition
// ============================================================================
// Job lists by slice size: slices of <= kTinyCap ids from the front of
// `small` (count ctr[kCtrJobs0]), slices of <= kSmallCap ids from its back
// (small[cap - 1 - k], count ctr[kCtrSmall]), larger ones in `big`
// (ctr[kCtrJobs1]), each with the first of its tiles (tile_off, their number
// in ctr[kCtrTiles]; any order of the slices does).  Slices of 0 or 1 ids are
// sorted already.  The batch's total goes to ctr[kCtrTotal]; more than ids_cap
// ids set bit 2 of ctr[kCtrOverflow], empty the write pass's item list and
// list nothing.  small == nullptr: no lists.
__global__ void k_classify(const unsigned long long* __restrict__ offsets, uint32_t q, Job* small, size_t cap,
                           Job* big, uint32_t* tile_off, uint32_t* ctr, unsigned long long ids_cap,
                           uint32_t* item_count, unsigned long long* big_ids) {
  const unsigned long long total = offsets[q];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *reinterpret_cast<unsigned long long*>(ctr + kCtrTotal) = total;
    if (total > ids_cap) {
      atomicOr(ctr + kCtrOverflow, 2u);
      if (item_count) *item_count = 0;
    }
  }
  if (!small || total > ids_cap) return;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < q; i += gridDim.x * blockDim.x) {
    const unsigned long long off = offsets[i];
    const unsigned long long sz = offsets[i + 1] - off;
    if (sz <= 1) continue;
    Job j;
    j.off = off;
    j.size = (uint32_t)sz;
    j.q = i;
    if (sz <= kTinyCap) {
      small[atomicAdd(ctr + kCtrJobs0, 1u)] = j;
    } else if (sz <= kSmallCap) {
      small[cap - 1 - atomicAdd(ctr + kCtrSmall, 1u)] = j;
    } else {
      const uint32_t at = atomicAdd(ctr + kCtrJobs1, 1u);
      big[at] = j;
      tile_off[at] = atomicAdd(ctr + kCtrTiles, (uint32_t)((sz + kTile - 1) / kTile));
      if (big_ids) atomicAdd(big_ids, sz);
    }
  }
}

// tile -> job
__global__ void k_tile_map(const Job* __restrict__ jobs, const uint32_t* __restrict__ tile_off,
                           const uint32_t* __restrict__ njobs_p, uint32_t* map) {
  const uint32_t njobs = *njobs_p;
  for (uint32_t j = blockIdx.x; j < njobs; j += gridDim.x) {
    const uint32_t t0 = tile_off[j], nt = (jobs[j].size + kTile - 1) / kTile;
    for (uint32_t k = threadIdx.x; k < nt; k += blockDim.x) map[t0 + k] = j;
  }
}

// Window histogram of every tile -> whist[job * G + window].
__global__ void __launch_bounds__(kTileThreads) k_win_hist(const Job* __restrict__ jobs,
                                                           const uint32_t* __restrict__ map,
                                                           const uint32_t* __restrict__ tile_off,
                                                           const uint32_t* __restrict__ ntiles_p, const int32_t* __restrict__ src,
                                                           uint32_t G, uint32_t wbits, uint32_t* whist) {
  const uint32_t ntiles = *ntiles_p;
  extern __shared__ uint32_t h[];  // [G]
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    for (uint32_t w = threadIdx.x; w < G; w += kTileThreads) h[w] = 0;
    __syncthreads();
    const uint32_t j = map[t];
    const Job jb = jobs[j];
    const uint32_t b0 = (t - tile_off[j]) * kTile;
    const uint32_t b1 = min(b0 + kTile, jb.size);
    uint32_t v[kTile / kTileThreads];
#pragma unroll
    for (uint32_t k = 0; k < kTile / kTileThreads; ++k) {
      const uint32_t i = b0 + k * kTileThreads + threadIdx.x;
      v[k] = (i < b1) ? (uint32_t)__ldcs(src + jb.off + i) : 0xffffffffu;
    }
#pragma unroll
    for (uint32_t k = 0; k < kTile / kTileThreads; ++k)
      if (v[k] != 0xffffffffu) atomicAdd(&h[v[k] >> wbits], 1u);
    __syncthreads();
    for (uint32_t w = threadIdx.x; w < G; w += kTileThreads)
      if (h[w]) atomicAdd(&whist[(size_t)j * G + w], h[w]);
    __syncthreads();
  }
}

// Per job: exclusive scan over its G window counts -> bases and cursors.
// With qwhist (the write pass's per-(query, window) counts) the job's counts
// are read from its query's row and copied to whist for k_win_sort.
__global__ void __launch_bounds__(kTileThreads) k_win_scan(const Job* __restrict__ jobs,
                                                           const uint32_t* __restrict__ njobs_p,
                                                           uint32_t G, uint32_t* __restrict__ whist,
                                                           const uint32_t* __restrict__ qwhist,
                                                           unsigned long long* wbase,
                                                           unsigned long long* wcur) {
  const uint32_t njobs = *njobs_p;
  __shared__ uint32_t wt[kTileWarps];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t per = (G + kTileThreads - 1) / kTileThreads;
  for (uint32_t j = blockIdx.x; j < njobs; j += gridDim.x) {
    const size_t base = (size_t)j * G;
    const uint32_t w0 = threadIdx.x * per;
    if (qwhist) {
      const size_t qbase = (size_t)jobs[j].q * G;
      for (uint32_t k = 0; k < per; ++k)
        if (w0 + k < G) whist[base + w0 + k] = qwhist[qbase + w0 + k];
    }
    uint32_t s = 0;
    for (uint32_t k = 0; k < per; ++k)
      if (w0 + k < G) s += whist[base + w0 + k];
    uint32_t x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) wt[w] = x;
    __syncthreads();
    uint32_t before = 0;
    for (uint32_t k = 0; k < w; ++k) before += wt[k];
    unsigned long long run = jobs[j].off + before + x - s;
    for (uint32_t k = 0; k < per; ++k) {
      if (w0 + k < G) {
        wbase[base + w0 + k] = run;
        wcur[base + w0 + k] = run;
        run += whist[base + w0 + k];
      }
    }
    __syncthreads();
  }
}

// Each tile: regroup its ids by window in shared memory, reserve the window
// ranges with one atomic per nonempty window, write contiguous runs.  With
// G <= kPerWarpMaxG each warp counts into its own counters (the counter's
// old value is the id's slot among its warp's ids of that window); the
// order inside a window does not matter, the ranking orders it.
__global__ void __launch_bounds__(kTileThreads, kTileBlocks) k_win_scatter(const Job* __restrict__ jobs,
                                                              const uint32_t* __restrict__ map,
                                                              const uint32_t* __restrict__ tile_off,
                                                              const uint32_t* __restrict__ ntiles_p, const int32_t* __restrict__ src,
                                                              int32_t* __restrict__ dst, uint32_t G,
                                                              uint32_t wbits, unsigned long long* wcur) {
  const uint32_t ntiles = *ntiles_p;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t nw = (G <= kPerWarpMaxG) ? kTileWarps : 1u;  // counter sets
  unsigned long long* gstart = reinterpret_cast<unsigned long long*>(smem_raw);  // [G]
  uint32_t* cnt = reinterpret_cast<uint32_t*>(gstart + G);                     // [nw][G]
  uint32_t* stage = cnt + nw * G;                                               // [kTile]
  __shared__ uint32_t wt[kTileWarps];
  const uint32_t lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  uint32_t* cw = cnt + (nw == 1 ? 0u : wp) * G;
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    for (uint32_t w = threadIdx.x; w < nw * G; w += kTileThreads) cnt[w] = 0;
    __syncthreads();
    const uint32_t j = map[t];
    const Job jb = jobs[j];
    const uint32_t b0 = (t - tile_off[j]) * kTile;
    const uint32_t n = min(b0 + kTile, jb.size) - b0;
    uint32_t v[kTile / kTileThreads];
    uint32_t slot[kTile / kTileThreads];
#pragma unroll
    for (uint32_t k = 0; k < kTile / kTileThreads; ++k) {
      const uint32_t i = k * kTileThreads + threadIdx.x;
      v[k] = (i < n) ? (uint32_t)__ldcs(src + jb.off + b0 + i) : 0xffffffffu;
    }
#pragma unroll
    for (uint32_t k = 0; k < kTile / kTileThreads; ++k)
      slot[k] = (v[k] != 0xffffffffu) ? atomicAdd(&cw[v[k] >> wbits], 1u) : 0u;
    __syncthreads();
    // exclusive scan over (window, counter set) in window-major order
    const uint32_t per = (G + kTileThreads - 1) / kTileThreads;
    const uint32_t w0 = threadIdx.x * per;
    uint32_t s = 0;
    for (uint32_t k = 0; k < per; ++k)
      if (w0 + k < G)
        for (uint32_t q = 0; q < nw; ++q) s += cnt[q * G + w0 + k];
    uint32_t x = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) wt[wp] = x;
    __syncthreads();
    uint32_t run = x - s;
    for (uint32_t k = 0; k < wp; ++k) run += wt[k];
    for (uint32_t k = 0; k < per; ++k) {
      const uint32_t w = w0 + k;
      if (w < G) {
        uint32_t tot = 0;
        for (uint32_t q = 0; q < nw; ++q) {
          const uint32_t c = cnt[q * G + w];
          cnt[q * G + w] = run + tot;  // first slot of this counter set in the tile
          tot += c;
        }
        // output position of the tile's id at stage slot i of window w:
        // gstart[w] + i (the window's start minus its local base)
        if (tot) gstart[w] = atomicAdd(&wcur[(size_t)j * G + w], (unsigned long long)tot) - run;
        run += tot;
      }
    }
    __syncthreads();
#pragma unroll
    for (uint32_t k = 0; k < kTile / kTileThreads; ++k)
      if (v[k] != 0xffffffffu) stage[cw[v[k] >> wbits] + slot[k]] = v[k];
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += kTileThreads) {
      const uint32_t id = stage[i];
      const uint32_t w = id >> wbits;
      dst[gstart[w] + i] = (int32_t)id;
    }
    __syncthreads();
  }
}

// ============================================================================
// Window sort
// ============================================================================
template <uint32_t BITS>
struct RankSmem {
  uint64_t bar;                             // completion of the window's bulk prefetch
  uint64_t pad_;
  uint32_t bm[WinCfg<BITS>::kWords];        // one bit per possible id of the window
  // output ranks [0, kStage) of the window, rank r at stage[r + (off & 3)] so
  // that the stage and the output share their 16-byte alignment
  int32_t stage[WinCfg<BITS>::kStage + 4];
  // first ids of the next window, loaded ahead: id i of a window at offset
  // off is at pf[i + (off & 3)]
  int32_t pf[WinCfg<BITS>::kPrefetch + 4];
  uint32_t wsum[WinCfg<BITS>::kWarps];      // set bits in each warp's word range
};

// Shared -> global bulk copy (the TMA unit) of `bytes` (a multiple of 16,
// both addresses 16-byte aligned), tracked as a bulk async-group.
__device__ __forceinline__ void bulk_copy_s2g(void* gdst, const void* ssrc, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(gdst),
               "r"(static_cast<uint32_t>(__cvta_generic_to_shared(ssrc))), "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
}
// Until the issued bulk stores have read their shared-memory source.
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory"); }
// Until the issued bulk stores are complete.
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }
// Generic-proxy writes to shared memory before async-proxy reads of them.
__device__ __forceinline__ void fence_proxy_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// Bit position of the highest set bit of x (x != 0).
__device__ __forceinline__ uint32_t bfind32(uint32_t x) {
  uint32_t b;
  asm("bfind.u32 %0, %1;" : "=r"(b) : "r"(x));
  return b;
}

// Position of bitmap word w in shared memory (see k_win_sort).
template <uint32_t BITS>
__device__ __forceinline__ uint32_t bm_at(uint32_t w) {
  return (w % WinCfg<BITS>::kLaneWords) * WinCfg<BITS>::kThreads + w / WinCfg<BITS>::kLaneWords;
}

// Persistent CTAs over the listed (job, window) pairs g = job * G + window
// (the windows of more than kWinWarpMax ids).
//   1. every id of window g (read from src, the scratch buffer) sets its bit
//      in a bitmap of the window's 2^wbits possible ids; its first kPrefetch
//      ids were brought into shared memory by a bulk copy (the TMA unit)
//      while the previous window ran;
//   2. every thread owns kLaneWords bitmap words: it counts their set bits,
//      takes its exclusive prefix over the CTA (warp scan + warp sums), i.e.
//      its ranks [pos, pos + cnt), then walks its nonzero words from the
//      highest down and emits the id of every set bit from its highest rank
//      down (bfind finds the highest set bit in one instruction), clearing
//      each word it read; ranks below kStage go to a shared-memory stage,
//      larger ones straight to the output;
//   3. the stage leaves by one bulk store (its 16-byte-aligned middle) and a
//      few plain stores (the ends).
// Warp 0 alone issues the next window's prefetch and the copy-out (their
// 64-bit offset arithmetic is per CTA, not per thread).  Three CTA barriers
// per window: bitmap complete, warp sums ready, stage complete (which also
// orders the bitmap's clearing before the next window's bits).  The ids of a
// window are distinct, so the set bits are the window's ids and their
// enumeration in bit order is the window in ascending order.  G is a power
// of two.
template <uint32_t BITS>
__global__ void __launch_bounds__(WinCfg<BITS>::kThreads, WinCfg<BITS>::kBlocks)
    k_win_sort(const uint32_t* __restrict__ list, const uint32_t* __restrict__ nlist_p, uint32_t G, uint32_t wbits,
               const uint32_t* __restrict__ whist, const unsigned long long* __restrict__ wbase,
               const int32_t* __restrict__ src, int32_t* __restrict__ out, uint32_t* err) {
  using C = WinCfg<BITS>;
  constexpr uint32_t kRankThreads = C::kThreads;
  constexpr uint32_t kRankWarps = C::kWarps;
  constexpr uint32_t kBmWords = C::kWords;
  constexpr uint32_t kStage = C::kStage;
  constexpr uint32_t kPrefetch = C::kPrefetch;
  launch_dependents();  // k_win_sort_warp, when all of these CTAs are here
  const uint32_t total = *nlist_p;  // listed (job, window) pairs
  extern __shared__ __align__(16) unsigned char smem_raw[];
  RankSmem<BITS>& s = *reinterpret_cast<RankSmem<BITS>*>(smem_raw);
  const uint32_t tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  uint4* bm4 = reinterpret_cast<uint4*>(s.bm);
  const uint32_t nwords = (1u << wbits) >> 5;   // 12 <= wbits <= BITS
  constexpr uint32_t kLaneWords = C::kLaneWords;
  const uint32_t tw0 = tid * kLaneWords;        // this thread's words [tw0, tw0 + kLaneWords)
  const bool owner = tw0 < nwords;
  // Word w of the bitmap (thread w / kLaneWords's word w % kLaneWords) is
  // stored at bm_at(w) = (w % kLaneWords) * kRankThreads + w / kLaneWords, so
  // that the lanes of a warp reading or clearing one word each of their own
  // ranges always hit 32 distinct banks.
  for (uint32_t i = tid; i < kBmWords / 4; i += kRankThreads) bm4[i] = make_uint4(0, 0, 0, 0);
  if (tid == 0) {
    mbar_init(&s.bar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  // The first kPrefetch ids of window g + gridDim.x are copied into s.pf
  // while window g is enumerated: their 16-byte-aligned middle [a0, a1) by
  // one bulk copy (thread 0, completing on s.bar, one barrier phase per
  // window even when it is empty); the up to 3 + 3 ids around it are loaded
  // into registers by threads 0..5 and written to s.pf by store_edge.  Every
  // thread waits on s.bar itself, so the bulk part needs no CTA barrier.
  auto prefetch_range = [&](unsigned long long o, uint32_t sz, unsigned long long* a0,
                            unsigned long long* a1) {
    const uint32_t n = sz < kPrefetch ? sz : kPrefetch;
    *a0 = (o + 3) & ~3ull;
    *a1 = (o + n) & ~3ull;
    if (*a1 < *a0) *a1 = *a0;
  };
  // The up to 3 + 3 ids around the bulk part: threads 0..5 load one each
  // into a register when the prefetch is issued and store it into s.pf only
  // before the window's last barrier, so the load's latency is hidden behind
  // the enumeration.
  int32_t edge_v = 0;
  int32_t edge_at = -1;  // s.pf slot of this thread's edge id, -1: none
  auto prefetch = [&](unsigned long long o, uint32_t sz) {
    unsigned long long a0, a1;
    prefetch_range(o, sz, &a0, &a1);
    const unsigned long long al = o & ~3ull;
    if (tid == 0) {
      mbar_arrive_expect_tx(&s.bar, (uint32_t)(a1 - a0) * 4u);
      if (a1 > a0) bulk_copy_g2s(&s.pf[a0 - al], src + a0, (uint32_t)(a1 - a0) * 4u, &s.bar);
    }
    const unsigned long long end = o + (sz < kPrefetch ? sz : kPrefetch);
    const unsigned long long h1 = a0 < end ? a0 : end;          // head [o, h1)
    const unsigned long long t0 = a1 > h1 ? a1 : h1;            // tail [t0, end)
    unsigned long long e = ~0ull;
    if (tid < 3 && o + tid < h1) e = o + tid;
    else if (tid >= 3 && tid < 6 && t0 + (tid - 3) < end) e = t0 + (tid - 3);
    edge_at = -1;
    if (e != ~0ull) {
      edge_v = __ldcs(src + e);
      edge_at = (int32_t)(e - al);
    }
  };
  auto store_edge = [&]() {
    if (edge_at >= 0) s.pf[edge_at] = edge_v;
    edge_at = -1;
  };
  uint32_t phase = 0;
  uint32_t size = 0;
  unsigned long long off = 0;
  if (blockIdx.x < total) {
    const uint32_t g0 = list[blockIdx.x];
    size = whist[g0];
    off = wbase[g0];
    if (wp == 0) prefetch(off, size);
  }
  store_edge();
  __syncthreads();
  for (uint32_t li = blockIdx.x; li < total; li += gridDim.x) {
    const uint32_t g = list[li];
    const uint32_t ln = li + gridDim.x;  // this CTA's next listed window
    uint32_t nsize = 0;
    unsigned long long noff = 0;
    if (ln < total) {
      const uint32_t gn = list[ln];
      nsize = whist[gn];
      noff = wbase[gn];
    }
    const int32_t* in = src + off;
    int32_t* dst = out + off;
    const uint32_t lo = (g & (G - 1)) << wbits;
    const uint32_t sh = (uint32_t)(off & 3);  // 16-byte alignment offset of this window's ids
    // this window's prefetched ids (every thread waits itself; the bitmap
    // was cleared and the stage written before the previous window's last
    // barrier), and the stage free of the previous window's bulk store
    const bool ok = mbar_wait_bounded(&s.bar, phase);
    phase ^= 1u;
    if (tid == 0) bulk_wait_read();
    // 1. set one bit per id: the prefetched ones from shared memory, the
    //    rest in rounds whose loads are all issued before the first atomic
    if (size >= 2 && ok) {
      const uint32_t npf = size < kPrefetch ? size : kPrefetch;
      for (uint32_t i = tid; i < npf; i += kRankThreads) {
        const uint32_t x = (uint32_t)s.pf[i + sh] - lo;
        atomicOr(&s.bm[bm_at<BITS>(x >> 5)], 1u << (x & 31));
      }
      for (uint32_t i0 = kPrefetch; i0 < size; i0 += kBatch * kRankThreads) {
        uint32_t a[kBatch];
#pragma unroll
        for (uint32_t k = 0; k < kBatch; ++k) {
          const uint32_t i = i0 + k * kRankThreads + tid;
          a[k] = kNone;
          if (i0 + k * kRankThreads + (wp << 5) < size && i < size) a[k] = (uint32_t)__ldcs(in + i) - lo;
        }
#pragma unroll
        for (uint32_t k = 0; k < kBatch; ++k)
          if (i0 + k * kRankThreads + (wp << 5) < size && a[k] != kNone)
            atomicOr(&s.bm[bm_at<BITS>(a[k] >> 5)], 1u << (a[k] & 31));
      }
    } else if (size == 1 && tid == 0) {
      dst[0] = s.pf[sh];
    }
    if (__syncthreads_or(!ok)) {  // bitmap complete; s.pf free
      // a bulk copy did not complete in time: flag it and stop (the results
      // are invalid); wait once more, again bounded, for that copy
      if (tid == 0) atomicOr(err, 1u);
      mbar_wait_bounded(&s.bar, phase ^ 1u);
      break;
    }
    if (ln < total && wp == 0) prefetch(noff, nsize);
    if (size < 2) {
      store_edge();
      __syncthreads();  // the next window's edge ids are in place
      size = nsize;
      off = noff;
      continue;  // uniform over the CTA
    }
    // 2a. set bits and nonzero words of this thread's range
    uint32_t cnt = 0, nz = 0;
    if (owner) {
#pragma unroll
      for (uint32_t k = 0; k < kLaneWords; ++k) {
        const uint32_t c = __popc(s.bm[k * kRankThreads + tid]);
        cnt += c;
        nz += min(c, 1u) << k;  // bit k: word k is nonzero
      }
    }
    uint32_t wtot;
    const uint32_t ex = warp_excl_sum(cnt, &wtot);
    if (lane == 0) s.wsum[wp] = wtot;
    __syncthreads();
    // 2b. enumerate the set bits in order
    const uint32_t ws = lane < kRankWarps ? s.wsum[lane] : 0u;
    uint32_t pos = __reduce_add_sync(0xffffffffu, lane < wp ? ws : 0u) + ex;
    // one iteration per set bit (a flat loop: a warp runs as many iterations
    // as its lane with the most bits), from rank pos + cnt - 1 down to pos;
    // the next lower nonzero word is fetched, and cleared, when the current
    // one is used up.  Ranks from kStage up go straight to the output, the
    // rest to the stage, in two loops so that no iteration tests the rank.
    uint32_t cur = 0, base = 0;
    const uint32_t base0 = lo + (tw0 << 5);  // id of bit 0 of this thread's first word
    uint32_t r = pos + cnt;
    const uint32_t split = max(pos, min(r, kStage));  // ranks >= split go straight out
    auto next_bit = [&]() -> uint32_t {
      if (cur == 0) {
        const uint32_t wi = bfind32(nz);
        nz ^= 1u << wi;
        cur = s.bm[wi * kRankThreads + tid];
        s.bm[wi * kRankThreads + tid] = 0u;
        base = base0 + (wi << 5);
      }
      const uint32_t b = bfind32(cur);
      cur ^= 1u << b;
      return base + b;
    };
    while (r > split) {
      const uint32_t id = next_bit();
      dst[--r] = (int32_t)id;
    }
    int32_t* st = s.stage + sh;
    while (r > pos) {
      const uint32_t id = next_bit();
      st[--r] = (int32_t)id;
    }
    store_edge();              // the next window's edge ids, before the last barrier
    fence_proxy_async_smem();  // the stage's writes before the bulk store reads them
    __syncthreads();
    // 3. staged ranks out (warp 0): the 16-byte-aligned middle by one bulk
    //    store, the up to 3 + 3 ids around it by plain stores; windows of
    //    fewer than 8 ids by plain stores
    const uint32_t ns = size < kStage ? size : kStage;
    if (wp == 0) {
      const unsigned long long al = off & ~3ull;
      const unsigned long long b0 = (off + 3) & ~3ull, b1 = (off + ns) & ~3ull;
      if (b1 > b0) {
        if (tid == 0) bulk_copy_s2g(out + b0, &s.stage[b0 - al], (uint32_t)(b1 - b0) * 4u);
        const uint32_t nh = (uint32_t)(b0 - off), nt = (uint32_t)(off + ns - b1);
        if (tid < nh) out[off + tid] = s.stage[sh + tid];
        else if (tid >= 4 && tid - 4 < nt) out[b1 + (tid - 4)] = s.stage[b1 - al + (tid - 4)];
      } else {
        for (uint32_t k = lane; k < ns; k += 32) dst[k] = s.stage[sh + k];
      }
    }
    size = nsize;
    off = noff;
  }
  if (tid == 0) bulk_wait_all();
}

}  // namespace

qcp_status ws_reserve_sort(qcp_index* ix, Workspace* ws, size_t jobs, size_t tiles);

// Blocks of k_win_scatter resident per SM with `smem` bytes of dynamic shared
// memory (its registers, not its shared memory, are the usual limit): the
// persistent grid is this many blocks per SM, so that no block waits for a
// second wave.
static uint32_t scatter_blocks_per_sm(size_t smem) {
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_win_scatter, kTileThreads, smem) != cudaSuccess || b < 1) {
    cudaGetLastError();
    b = 1;
  }
  return (uint32_t)b;
}

static uint32_t id_bits(uint64_t n) {
  uint32_t idbits = 1;
  while (idbits < 31 && (1ull << idbits) < n) ++idbits;
  return idbits;
}

// The window sort for 2^wbits-id windows (the instantiation whose bitmap
// holds them), over at most `max_pairs` (job, window) pairs.
template <uint32_t BITS>
static void launch_win_sort_t(uint64_t max_pairs, uint32_t sms, const uint32_t* list, const uint32_t* nlist,
                              uint32_t G, uint32_t wbits, const uint32_t* whist, const unsigned long long* wbase,
                              const int32_t* src, int32_t* out, uint32_t* err, cudaStream_t s) {
  using C = WinCfg<BITS>;
  // resident CTAs per SM from the occupancy API (its shared memory decides),
  // once per device and thread
  static thread_local int occ_dev = -1;
  static thread_local uint32_t occ = C::kBlocks;
  int dev = 0;
  if (cudaGetDevice(&dev) == cudaSuccess && dev != occ_dev) {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_win_sort<BITS>, C::kThreads, sizeof(RankSmem<BITS>)) ==
            cudaSuccess &&
        b > 0) {
      occ = (uint32_t)b;
      occ_dev = dev;
    } else {
      cudaGetLastError();
    }
  }
  const uint64_t cap = (uint64_t)sms * occ;
  const uint32_t grid = (uint32_t)(max_pairs < cap ? max_pairs : cap);
  if (grid)
    k_win_sort<BITS><<<grid, C::kThreads, sizeof(RankSmem<BITS>), s>>>(list, nlist, G, wbits, whist, wbase, src, out,
                                                                       err);
}

// The windows of a call: k_win_split lists them (counts in ctr[kCtrWinBig],
// ctr[kCtrWinSmall], zeroed by the caller), the bitmap sort takes the large
// ones and one warp each the small ones, beside it as soon as all of its CTAs are
// on the SMs (but not in a call that reports phase times).  On two streams
// either could come first, and where the small ones' did, CTAs of the bitmap
// sort waited for them with their full share of windows (10,000 boxes over 16 M
// points 7.65 ms one time and 9.6 the next; one after the other 7.75).  lists
// holds 2 * max_pairs entries; max_pairs bounds the (job, window) pairs.
static qcp_status launch_win_sort(Workspace* ws, uint64_t max_pairs, uint32_t sms, const uint32_t* njobs, uint32_t G,
                                  uint32_t wbits, const uint32_t* whist, const unsigned long long* wbase, uint32_t* lists,
                                  uint32_t* ctr, const int32_t* src, int32_t* out, uint32_t* err, cudaStream_t s,
                                  bool stats) {
  uint32_t* big = lists;
  uint32_t* small = lists + max_pairs;
  const uint64_t split_blocks = (max_pairs + 255) / 256;
  k_win_split<<<(uint32_t)(split_blocks < (uint64_t)sms * 8 ? split_blocks : (uint64_t)sms * 8), 256, 0, s>>>(
      njobs, G, whist, big, ctr + kCtrWinBig, small, ctr + kCtrWinSmall,
      stats && ws->timing ? ws->d_stats + kStatBitmapIds : nullptr);
  if (wbits >= 18) launch_win_sort_t<18>(max_pairs, sms, big, ctr + kCtrWinBig, G, wbits, whist, wbase, src, out, err, s);
  else if (wbits == 17) launch_win_sort_t<17>(max_pairs, sms, big, ctr + kCtrWinBig, G, wbits, whist, wbase, src, out, err, s);
  else launch_win_sort_t<16>(max_pairs, sms, big, ctr + kCtrWinBig, G, wbits, whist, wbase, src, out, err, s);
  if (stats) mark(ws, kEvSortBitmap, s);
  const uint64_t warp_blocks = (max_pairs + kTinyWarps - 1) / kTinyWarps;
  const uint64_t warp_cap = (uint64_t)sms * kWinWarpBlocks;
  cudaLaunchAttribute beside{};
  beside.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  beside.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((uint32_t)(warp_blocks < warp_cap ? warp_blocks : warp_cap));
  cfg.blockDim = dim3(kTinyWarps * 32);
  cfg.dynamicSmemBytes = sizeof(TinySmem<kWinWarpMax>);
  cfg.stream = s;
  cfg.attrs = &beside;
  cfg.numAttrs = ws->timing || max_pairs == 0 ? 0 : 1;  // (no pairs: the kernel before it is not k_win_sort)
  QCP_CUDA(cudaLaunchKernelEx(&cfg, k_win_sort_warp, (const uint32_t*)small, (const uint32_t*)(ctr + kCtrWinSmall), G,
                              wbits, whist, wbase, src, out));
  return QCP_OK;
}

static qcp_status set_sort_attrs(const qcp_index* ix, size_t scatter_max) {
  static thread_local int attrs_device = -1;  // attributes are per device
  if (attrs_device != ix->device) {
    QCP_CUDA(cudaFuncSetAttribute(k_sort_small, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(BucketSmem)));
    QCP_CUDA(cudaFuncSetAttribute(k_sort_tiny, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(TinySmem<kTinyCap>)));
    QCP_CUDA(cudaFuncSetAttribute(k_win_sort_warp, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(TinySmem<kWinWarpMax>)));
    QCP_CUDA(cudaFuncSetAttribute(k_win_sort<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(RankSmem<16>)));
    QCP_CUDA(cudaFuncSetAttribute(k_win_sort<17>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(RankSmem<17>)));
    QCP_CUDA(cudaFuncSetAttribute(k_win_sort<18>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(RankSmem<18>)));
    QCP_CUDA(cudaFuncSetAttribute(k_win_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)scatter_max));
    attrs_device = ix->device;
  }
  return QCP_OK;
}

qcp_status classify_slices(qcp_index* ix, Workspace* ws, uint32_t q, bool sort, uint64_t cap, uint32_t* item_count,
                           cudaStream_t s) {
  if (sort) QCP_TRY(ws_reserve_sort(ix, ws, (size_t)q + 256, 0));
  k_classify<<<(q + 255) / 256, 256, 0, s>>>((const unsigned long long*)ws->offsets, q,
                                             sort ? reinterpret_cast<Job*>(ws->jobs[0]) : nullptr, ws->jobs_cap,
                                             reinterpret_cast<Job*>(ws->jobs[1]), ws->job_tiles, ws->ctr, cap,
                                             item_count, ws->timing ? ws->d_stats + kStatWindowIds : nullptr);
  note_launch();
  return check_launch("k_classify");
}

// The tables of the window partition for at most njobs slices: counts (u32),
// bases and cursors (u64) per (slice, window), and the two window lists.
struct SortTables {
  uint32_t* whist;
  unsigned long long *wbase, *wcur;
  uint32_t* lists;
  size_t bytes;
  SortTables(void* p, size_t njobs, uint32_t G) {
    const size_t nw = njobs * G;
    const size_t hist_bytes = (nw * 4 + 15) & ~(size_t)15;
    char* c = static_cast<char*>(p);
    whist = reinterpret_cast<uint32_t*>(c);
    wbase = reinterpret_cast<unsigned long long*>(c + hist_bytes);
    wcur = wbase + nw;
    lists = reinterpret_cast<uint32_t*>(wcur + nw);  // 2 * nw
    bytes = hist_bytes + nw * 24 + 64;
  }
};

// The windows of the larger slices: partition and sort, over at most njobs
// slices and ntiles tiles.  stats: a call that reports phase times.
static qcp_status sort_windows(qcp_index* ix, Workspace* ws, size_t njobs, uint64_t ntiles, const SortTables& t,
                               uint32_t G, uint32_t wbits, cudaStream_t s, bool stats) {
  const uint32_t sms = (uint32_t)num_sms();
  const uint32_t nsets = (G <= kPerWarpMaxG) ? kTileWarps : 1u;
  const size_t scatter_bytes = (size_t)G * (8 + 4 * nsets) + kTile * 4;
  const size_t nw = njobs * G;
  uint32_t* ctr = ws->ctr;
  const Job* big = reinterpret_cast<const Job*>(ws->jobs[1]);
  auto at_most = [](uint64_t a, uint64_t b) { return (uint32_t)(a < b ? a : b); };
  k_tile_map<<<at_most(njobs, sms * 8), 256, 0, s>>>(big, ws->job_tiles, ctr + kCtrJobs1, ws->seg_hist);
  // per-(job, window) counts: from the write pass when it gathered them
  const bool have_counts = ws->hist_G == G && ws->hist_bits == wbits;
  if (!have_counts) {
    QCP_CUDA(cudaMemsetAsync(t.whist, 0, sizeof(uint32_t) * nw, s));
    k_win_hist<<<at_most(ntiles, sms * 8), kTileThreads, sizeof(uint32_t) * G, s>>>(
        big, ws->seg_hist, ws->job_tiles, ctr + kCtrTiles, ws->out_ids, G, wbits, t.whist);
    note_launch();
  }
  k_win_scan<<<at_most(njobs, sms * 16), kTileThreads, 0, s>>>(big, ctr + kCtrJobs1, G, t.whist,
                                                               have_counts ? ws->qwhist : nullptr, t.wbase, t.wcur);
  k_win_scatter<<<at_most(ntiles, sms * scatter_blocks_per_sm(scatter_bytes)), kTileThreads, scatter_bytes, s>>>(
      big, ws->seg_hist, ws->job_tiles, ctr + kCtrTiles, ws->out_ids, ws->tmp_ids, G, wbits, t.wcur);
  if (stats) {
    mark(ws, kEvSortPart, s);
    ws->sort_part_marked = ws->timing;
  }
  // (the window lists' counters are zero since the call's start)
  QCP_TRY(launch_win_sort(ws, nw, sms, ctr + kCtrJobs1, G, wbits, t.whist, t.wbase, t.lists, ctr, ws->tmp_ids,
                          ws->out_ids, ctr + kCtrTimeout, s, stats));
  note_launch(6);
  return check_launch("segmented sort windows");
}

static constexpr size_t kScatterMax = (size_t)(1u << (31 - kWinBits)) * 16 + kTile * 4;

qcp_status segmented_sort(qcp_index* ix, Workspace* ws, cudaStream_t s) {
  ws->sort_part_marked = false;
  const uint32_t idbits = id_bits(ix->n);
  const uint32_t sms = (uint32_t)num_sms();
  QCP_TRY(set_sort_attrs(ix, kScatterMax));
  uint32_t* ctr = ws->ctr;
  Job* small = reinterpret_cast<Job*>(ws->jobs[0]);
  const uint32_t ntiny = ws->h_ctr[kCtrJobs0];
  const uint32_t nsmall = ws->h_ctr[kCtrSmall];
  const uint32_t nbig = ws->h_ctr[kCtrJobs1];
  ws->sort_small_jobs = ntiny + nsmall;
  ws->sort_msd_jobs = nbig;
  // slices of two classes: the smaller ones' kernel beside the other's (not in a
  // call that reports phase times); each leaves much of the chip idle in a
  // batch of some hundred boxes (1,000 over 2 M points 314 -> 261 us) and its
  // tail in large ones (10,000 over 16 M points 8,024 -> 7,954)
  const bool fork = !ws->timing && (nbig ? ntiny + nsmall : (ntiny && nsmall));
  if (fork) QCP_TRY(ws_reserve_side(ws));
  cudaStream_t tiny_s = fork ? ws->side : s, small_s = fork && nbig ? ws->side : s;
  if (fork) QCP_CUDA(ws_branch(ws, 2, s, ws->side));
  if (ntiny) {
    k_sort_tiny<<<min((ntiny + kTinyWarps - 1) / kTinyWarps, sms * kTinyBlocks), kTinyWarps * 32,
                  sizeof(TinySmem<kTinyCap>), tiny_s>>>(small, ctr + kCtrJobs0, ws->out_ids, idbits);
    note_launch();
    QCP_TRY(check_launch("k_sort_tiny"));
  }
  if (nsmall) {
    k_sort_small<<<min(nsmall, sms * 4), kSmallThreads, sizeof(BucketSmem), small_s>>>(
        small + ws->jobs_cap, ctr + kCtrSmall, ws->out_ids, idbits);
    note_launch();
    QCP_TRY(check_launch("k_sort_small"));
  }
  mark(ws, kEvSortSmall, s);
  if (nbig == 0) {
    if (fork) QCP_CUDA(ws_branch(ws, 4, ws->side, s));
    return QCP_OK;
  }
  uint32_t wbits = 0, G = 0;
  sort_window_shape(ix, ws, &wbits, &G);
  const uint32_t ntiles = ws->h_ctr[kCtrTiles];
  QCP_TRY(ws_reserve_sort(ix, ws, 0, ntiles));
  QCP_TRY(ws_reserve_tables(ws, SortTables(nullptr, nbig, G).bytes));
  QCP_TRY(sort_windows(ix, ws, nbig, ntiles, SortTables(ws->tables, nbig, G), G, wbits, s, true));
  if (fork) QCP_CUDA(ws_branch(ws, 4, ws->side, s));
  return QCP_OK;
}


// Window bits and window count of a call (ws->win_bits, bounded as in
// segmented_sort).
void sort_window_shape(const qcp_index* ix, const Workspace* ws, uint32_t* wbits, uint32_t* G);
static void window_shape(const qcp_index* ix, const Workspace* ws, uint32_t* wbits, uint32_t* G) {
  const uint32_t idbits = id_bits(ix->n);
  uint32_t wb = ws->win_bits ? ws->win_bits : kDefaultWinBits;
  if (wb > kWinBits) wb = kWinBits;
  if (idbits > 13 && wb < idbits - 13) wb = idbits - 13;
  *wbits = idbits < wb ? idbits : wb;
  *G = 1u << (idbits - *wbits);
}

void sort_window_shape(const qcp_index* ix, const Workspace* ws, uint32_t* wbits, uint32_t* G) {
  window_shape(ix, ws, wbits, G);
}

// Bytes of the per-(job, window) tables that segmented_sort_device needs for
// q queries with ws's window bits.
size_t sort_tables_bytes(const qcp_index* ix, const Workspace* ws, uint32_t q) {
  uint32_t wbits = 0, G = 0;
  window_shape(ix, ws, &wbits, &G);
  return SortTables(nullptr, q, G).bytes;
}

// segmented_sort without host readbacks, for at most max_ids ids: job and tile
// counts stay on the device, every launch has a fixed grid and the kernels
// read the counts.  The slices that single CTAs and warps sort run on ws->side
// beside the window partition and the bitmap sort: each of the kernels leaves
// most of the chip idle on a plan's small batch (a run of 64 boxes on 16 M
// points, 62 us of it sort kernels: 194 -> 153 us with this branch and the tiles
// numbered by k_classify instead of a scan; 143 with the small windows behind
// the bitmap sort's start instead of on the branch).
// Tables (sort_tables_bytes) and the tile map (at least
// max_ids / kSortTile + q entries, ws->seg_hist) are the caller's.
// Stream-capturable.
qcp_status segmented_sort_device(qcp_index* ix, Workspace* ws, uint32_t q, void* tables, cudaStream_t s) {
  if (q == 0) return QCP_OK;
  const uint32_t idbits = id_bits(ix->n);
  uint32_t wbits = 0, G = 0;
  window_shape(ix, ws, &wbits, &G);
  const uint32_t sms = (uint32_t)num_sms();
  QCP_TRY(set_sort_attrs(ix, kScatterMax));
  uint32_t* ctr = ws->ctr;
  Job* small = reinterpret_cast<Job*>(ws->jobs[0]);
  QCP_CUDA(ws_branch(ws, 2, s, ws->side));
  k_sort_tiny<<<sms * kTinyBlocks, kTinyWarps * 32, sizeof(TinySmem<kTinyCap>), ws->side>>>(
      small, ctr + kCtrJobs0, ws->out_ids, idbits);
  k_sort_small<<<sms * 4, kSmallThreads, sizeof(BucketSmem), ws->side>>>(small + ws->jobs_cap, ctr + kCtrSmall,
                                                                         ws->out_ids, idbits);
  note_launch(2);
  QCP_TRY(sort_windows(ix, ws, q, ~0ull, SortTables(tables, q, G), G, wbits, s, false));
  QCP_CUDA(ws_branch(ws, 4, ws->side, s));
  return QCP_OK;
}

}  // namespace qcp
