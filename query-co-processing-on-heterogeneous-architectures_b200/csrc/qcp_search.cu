// Range-search traversal kernels.
//
// Batched pipeline (QCP_ALGO_BATCHED), for the whole query batch at once:
//   1. k_expand, once per level above the leaves' parents: every
//      (query, node) item of level l becomes the (query, child) items of the
//      children whose MBR overlaps the query (warp per item, ballot
//      compaction, one atomic per 32 items written).
//   2. the (query, level-1 node) items are counted.  k_join, for large batches,
//      which are ordered by node first (k_node_hist, a scan, k_node_scatter):
//      one CTA per run of items, the queries' boxes in shared memory, the
//      node's leaf MBRs in registers, and each partially covered leaf that some
//      box of the run overlaps loaded once and tested against all of them.
//      k_count, for the others: a warp per item or per 32-leaf group of one.
//      Both count leaves whose MBR lies inside a box without touching their
//      objects (unless the index holds a rectangle with lo > hi).
//   3. exclusive scan of the per-query counts -> CSR offsets.
//   4. k_leafwrite: a warp per item reserves its item's slice of the query's
//      output with one atomic and writes ids (whole id runs for covered
//      leaves, the hit bits k_join recorded, or a test of the leaf's objects).
//   5. per-query sort of the ids (qcp_segsort.cu).
//
// Plain traversal (QCP_ALGO_PLAIN): k_mprs, one query per CUDA block as the
// reference's global_RestartScanning_and_ParentCheck
// (src/tree/mphr.cpp:303-438), but depth first over the implicit node layout
// with the path's overlap masks in shared memory instead of a restart from the
// root after every run of leaves; run twice (count, then write).
//
// The hit predicate everywhere is the reference's closed-interval test
// (src/node/node_soa.cpp:94-113).
#include <algorithm>
#include <cfloat>
#include <cstring>
#include <thread>

#include "qcp_internal.cuh"
#include "qcp_tree.cuh"

namespace qcp {

namespace {

// ---------------------------------------------------------------------------
// Batched pipeline kernels
// ---------------------------------------------------------------------------
__global__ void k_init_items(uint2* items, uint32_t q, uint32_t node, uint32_t* count) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < q; i += gridDim.x * blockDim.x)
    items[i] = make_uint2(i, node);
  if (blockIdx.x == 0 && threadIdx.x == 0) *count = q;
}

// LPI lanes per (query, node) item (32, 16 or 8: 1, 2 or 4 items per warp
// at once); each group tests its item's children LPI at a time and the
// overlapping ones are compacted with one warp ballot into the warp's stage in
// shared memory, which leaves 32 items at a time.  One atomic per round on
// the output counter bound the kernel (100,000 queries over 64 M points: 250,000
// atomics on one address, 152 us); one per 32 items takes 63 us.
// in == nullptr: the root level, item i is (i, node 0).
template <int D, int LPI>
__global__ void __launch_bounds__(256) k_expand(const float* __restrict__ boxes,
                                                const uint2* __restrict__ in,
                                                const uint32_t* __restrict__ in_count, uint32_t nroot,
                                                uint2* __restrict__ out, uint32_t* out_count,
                                                uint64_t out_cap, const float* __restrict__ child_mbr,
                                                uint64_t nchild, uint64_t child_pad, uint32_t fanout,
                                                uint32_t* overflow, uint32_t* need) {
  constexpr uint32_t kGroups = 32 / LPI;
  __shared__ uint2 stage_all[8][64];
  const uint32_t lane = threadIdx.x & 31;
  uint2* stage = stage_all[threadIdx.x >> 5];
  const uint32_t grp = lane / LPI, gl = lane % LPI;
  // the counter keeps counting past the capacity when a level overflowed
  const uint32_t nin = in ? (uint32_t)min((uint64_t)*in_count, out_cap) : nroot;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  const uint32_t rounds = (fanout + LPI - 1) / LPI;  // warp-uniform
  uint32_t held = 0;                                 // staged items (warp-uniform)
  auto flush = [&](uint32_t k) {                     // the first k <= 32 staged items out
    __syncwarp();
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(out_count, k);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (lane < k) {
      const uint64_t pos = (uint64_t)base + lane;
      if (pos < out_cap) out[pos] = stage[lane];
      else atomicOr(overflow, 1u);
    }
    if (lane == 0 && (uint64_t)base + k > out_cap) atomicMax(need, base + k);
    // the rest (fewer than 32) to the front
    const uint2 rest = stage[32 + lane];
    __syncwarp();
    stage[lane] = rest;
    held -= k;
    __syncwarp();
  };
  for (uint32_t i0 = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kGroups; i0 < nin; i0 += warps * kGroups) {
    const uint32_t i = i0 + grp;
    const bool have = i < nin;
    uint2 it = make_uint2(0, 0);
    Box<D> b;
    uint64_t c0 = 0, c1 = 0;
    if (have) {
      it = in ? in[i] : make_uint2(i, 0);
      b = load_box<D>(boxes, it.x);
      c0 = (uint64_t)it.y * fanout;
      c1 = (c0 + fanout < nchild) ? c0 + fanout : nchild;
    }
    for (uint32_t r = 0; r < rounds; ++r) {
      const uint64_t c = c0 + (uint64_t)r * LPI + gl;
      bool ov = false, in_ = false;
      if (have && c < c1) test_node<D>(b, child_mbr, child_pad, c, ov, in_);
      const uint32_t wm = __ballot_sync(0xffffffffu, ov);
      if (!wm) continue;  // warp-uniform
      if (ov) stage[held + __popc(wm & lane_lt_mask())] = make_uint2(it.x, (uint32_t)c);
      held += __popc(wm);
      if (held >= 32) flush(32);
    }
  }
  if (held) flush(held);
}

// Items per node (of `nodes`) from which node order and k_join pay: the host
// knows only the queries, so the kernels decide from the item count whether
// the batch is ordered.  Below it a node's leaves are shared by too few items
// to pay for k_join's staging (4.8 M points, 2,400 boxes of four ids, 2 items
// per node: k_join 34 us, k_count 12); 16 M points, 1,900 boxes, 29 per node:
// 110 against 143, and 32 M 8-D rectangles, 3,000 boxes, 13 per node: 154
// against 202.  Nor with so few items in all that k_join's runs are short (3 M
// points, 2,314 boxes, 5,000 items: 34 against 12).
constexpr uint32_t kNodeOrderItems = 12, kNodeOrderMinItems = 24576;
__device__ __forceinline__ bool is_ordered(uint32_t nitems, uint64_t nodes) {
  return nodes && nitems >= kNodeOrderMinItems && nitems >= nodes * kNodeOrderItems;
}

// Items per level-1 node, and the items in node order (cursor: the exclusive
// sums of the counts, advanced in place) or, in a batch that is not ordered,
// as they are.
__global__ void k_node_hist(const uint2* __restrict__ items, const uint32_t* __restrict__ count, uint64_t cap,
                            uint64_t nodes, uint32_t* hist) {
  const uint32_t n = (uint32_t)min((uint64_t)*count, cap);
  if (!is_ordered(n, nodes)) return;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    atomicAdd(hist + items[i].y, 1u);
}

__global__ void k_node_scatter(const uint2* __restrict__ items, const uint32_t* __restrict__ count, uint64_t cap,
                               uint64_t nodes, uint32_t* cursor, uint2* __restrict__ out, uint32_t* out_count) {
  const uint32_t n = (uint32_t)min((uint64_t)*count, cap);
  const bool ordered = is_ordered(n, nodes);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint2 it = items[i];
    out[ordered ? atomicAdd(cursor + it.y, 1u) : i] = it;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) *out_count = n;
}

enum { kCount = 0, kWrite = 1 };  // modes of the plain traversal

// What the count pass hands to the write pass.  Per item and 32-leaf group,
// rec = {overlapping leaves, covered leaves, word offset of the hit bits of
// its partially covered leaves, hits}; per partially covered leaf and
// 128-object chunk 32 bytes in mask, bit k of byte l = object 4l + k is a hit.  The write pass then copies ids without testing a leaf MBR or a
// coordinate again.  A group whose hit bits did not fit (words past
// mask_cap), or that records none (mask == nullptr), is marked kNoMask and
// the write pass tests its partially covered leaves.  rec == nullptr: counts
// only.
struct HitCache {
  uint4* rec;                  // [item][F / 32]
  uint32_t* mask;              // hit bits
  uint32_t mask_cap;           // words
  unsigned long long* cursor;  // words asked for so far (may pass mask_cap)
};

constexpr uint32_t kChunkWords = 8;  // hit words of a 128-object chunk

// Four consecutive objects per lane in registers: a warp holds 128 objects of
// a leaf.
template <int D, bool RECT>
struct Quad {
  float lo[D][4], hi[RECT ? D : 1][4];
};
__device__ __forceinline__ void load_four(float (&v)[4], const float* p) {
  const float4 x = __ldg(reinterpret_cast<const float4*>(p));
  v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
}
template <int D, bool RECT>
__device__ __forceinline__ void load_quad(Quad<D, RECT>& c, const float* coords, uint64_t npad, uint64_t p) {
#pragma unroll
  for (int d = 0; d < D; ++d) {
    load_four(c.lo[d], coords + (uint64_t)d * npad + p);
    if constexpr (RECT) load_four(c.hi[d], coords + (uint64_t)(D + d) * npad + p);
  }
}

// The closed-interval test on sign bits: an object is a hit iff neither
// e.hi - q.lo nor q.hi - e.lo is negative in any dimension.  The rounded
// difference of two floats has the sign of the exact one (subnormals are not
// flushed); a difference of zeros is -0 only if both operands allow it, so a
// zero box bound is passed as +0 in -q.lo and q.hi; a NaN bound gives the
// canonical NaN, sign clear, and passes as the negated comparison does;
// objects are finite.  So this is overlaps1 exactly.  The differences go to
// the FMA pipe and one three-input logic operation per object and dimension
// collects the signs; comparisons would all be issued to the ALU pipe.
// s[v] |= (sign bit) object v misses in dimension d.
template <int D, bool RECT>
__device__ __forceinline__ void miss_dim(const Quad<D, RECT>& c, int d, float nlo, float hi, uint32_t (&s)[4]) {
#pragma unroll
  for (int v = 0; v < 4; ++v)
    s[v] |= __float_as_uint(__fadd_rn(RECT ? c.hi[RECT ? d : 0][v] : c.lo[d][v], nlo)) |
            __float_as_uint(__fsub_rn(hi, c.lo[d][v]));
}
// The signs of a and b as bytes 0 and 1 (0xff or 0; selector bit 3 replicates
// the selected byte's sign).
__device__ __forceinline__ uint32_t sign_bytes(uint32_t a, uint32_t b) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, 0x00fb;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
// Hit bits of four objects (bit v: the sign of s[v] is clear): the four signs
// as bytes, masked to 1, 2, 4, 8 and summed.
__device__ __forceinline__ uint32_t hit_bits(const uint32_t (&s)[4]) {
  const uint32_t m = __byte_perm(sign_bytes(s[0], s[1]), sign_bytes(s[2], s[3]), 0x5410);
  return __dp4a(~m & 0x08040201u, 0x01010101u, 0u);
}

// A box in shared memory: {-lo, hi} per dimension, zeros as +0.
template <int D>
struct BoxRow {
  float v[2 * D];  // -lo0, hi0, -lo1, hi1, ..
  __device__ __forceinline__ void load(const float* row) {
    if constexpr (D % 2 == 0) {
#pragma unroll
      for (int e = 0; e < 2 * D; e += 4)
        *reinterpret_cast<float4*>(v + e) = *reinterpret_cast<const float4*>(row + e);
    } else {
#pragma unroll
      for (int e = 0; e < 2 * D; e += 2)
        *reinterpret_cast<float2*>(v + e) = *reinterpret_cast<const float2*>(row + e);
    }
  }
};

// Items of one CTA's run at most: one per thread.
constexpr uint32_t kJoinItems = 128;
constexpr uint32_t kJoinThreads = 128;
constexpr uint32_t kJoinWarps = kJoinThreads / 32;
constexpr uint32_t kJoinTasks = 8;  // tasks per CTA in large batches
constexpr uint32_t kPairs = 8;      // (leaf, box) pairs counted and stored together

// Counts: qcount[q] of every query, and the records of hc.  A task is a run of
// consecutive items and one 32-leaf group of their nodes; the items of one
// node are treated together: the leaves' coordinates, which one warp per item
// read again for every item, are read once per run.  That read bounded the
// pass: 32 M 8-D rectangles, 50,000 boxes (426,542 items, 1.7 M partially
// covered leaves of 8 KB) 2.53 -> 0.82 ms; 16 M 3-D points, 10,000 boxes 0.68 ->
// 0.30 ms; 64 M 2-D points, 100,000 boxes 0.50 -> 0.25 ms.  The run length
// follows from the item count: kJoinTasks tasks per CTA (the tail of the last
// ones is short), at most kJoinItems items; small batches get one item per
// task, its leaves spread over the warps.
// What remains is bound by issue and by what shared memory can broadcast (a
// box of 2 D floats takes 2 D cycles of an SM whatever the width of the
// loads), so a (leaf, box) pair is kept short: four objects per lane, sign
// bits instead of comparisons, the leaf's boxes from a list, a byte of hit
// bits per lane instead of ballots, and the bytes of kPairs pairs are counted
// and stored together.  (Prefetching the next leaf, into registers or L2,
// measured 15 % slower; packed f32x2 differences need every bound twice and
// were slower too.)
template <int D, bool RECT>
__global__ void __launch_bounds__(kJoinThreads, (RECT ? 2 * D : D) > 8 ? 4 : ((RECT ? 2 * D : D) > 4 ? 6 : 8))
    k_join(TreeView t, const float* __restrict__ boxes, const uint2* __restrict__ items,
           const uint32_t* __restrict__ item_count, uint32_t* work, unsigned long long* qcount, uint64_t item_cap,
           uint64_t nodes, unsigned long long* stats, HitCache hc) {
  __shared__ __align__(16) float bx[kJoinItems * 2 * D];
  __shared__ uint2 item[kJoinItems];
  __shared__ uint32_t part[kJoinItems], cov[kJoinItems];    // partially covered and covered leaves
  __shared__ uint32_t hits[kJoinItems], moff[kJoinItems];   // moff kNoMask: no hit bits kept
  __shared__ uint16_t s_list[kJoinWarps][kJoinItems];       // the warp's leaf: items that overlap it
  __shared__ __align__(16) uint8_t s_hit[kJoinWarps][kPairs * 32];  // hit bits of kPairs pairs
  __shared__ uint32_t s_pair[kJoinWarps][kPairs];           // their item | leaf << 16 | chunk << 24
  __shared__ uint32_t s_task, s_any, s_wsum[kJoinWarps];
  __shared__ unsigned long long s_base;
  const uint32_t F = t.fanout, G = F >> 5;
  const uint32_t tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const uint32_t nitems = (uint32_t)min((uint64_t)*item_count, item_cap);
  if (!is_ordered(nitems, nodes)) return;  // k_count's
  const float* lmbr = t.mbr[0];
  const uint64_t lpad = t.pad[0], nleaves = t.nodes[0];
  const uint32_t chunks = (F + 127u) >> 7;  // 128-object chunks of a leaf
  const uint32_t wpl = chunks * kChunkWords;
  uint64_t want = (uint64_t)nitems * G / (gridDim.x * kJoinTasks);
  const uint32_t runlen = want < 1 ? 1u : (want > kJoinItems ? kJoinItems : (uint32_t)want);
  uint32_t n_cov = 0, n_part = 0;  // work counters of this thread's items
  unsigned long long o_cov = 0;
  uint16_t* list = s_list[wp];
  uint8_t* bytes = s_hit[wp];
  uint32_t* pairs = s_pair[wp];
  uint32_t fetched = 0;  // thread 0: the task after the current one
  if (tid == 0) s_task = atomicAdd(work, 1u);
  for (;;) {
    __syncthreads();  // the task is known, the previous one finished with the shared memory
    const uint32_t g = s_task % G;
    const uint64_t i0 = (uint64_t)(s_task / G) * runlen;
    if (i0 >= nitems) break;
    const uint32_t rn = (uint32_t)min((uint64_t)runlen, nitems - i0);
    if (tid < rn) item[tid] = items[i0 + tid];
    __syncthreads();
    if (tid == 0) fetched = atomicAdd(work, 1u);
    for (uint32_t a = 0; a < rn;) {
      // the run's next node and its items [a, a + m)
      const uint32_t node = item[a].y;
      uint32_t m = 0;
      for (uint32_t j = a; j < rn; j += 32) {
        const uint32_t diff = __ballot_sync(0xffffffffu, j + lane >= rn || item[j + lane].y != node);
        m += diff ? __ffs(diff) - 1 : 32;
        if (diff) break;
      }
      const uint64_t l0 = (uint64_t)node * F + g * 32;  // the group's first leaf
      const uint32_t nl = l0 < nleaves ? (uint32_t)min((uint64_t)32, nleaves - l0) : 0u;
      for (uint32_t e = tid; e < m * 2 * D; e += kJoinThreads) {
        const uint32_t j = e / (2 * D), c = e % (2 * D);
        const float v = __ldg(boxes + (uint64_t)item[a + j].x * (2 * D) + c);
        bx[j * 2 * D + (c < D ? 2 * c : 2 * (c - D) + 1)] = v == 0.f ? 0.f : (c < D ? -v : v);
      }
      if (tid == 0) s_any = 0;
      __syncthreads();
      // A. every item's masks: a leaf's MBR per lane in registers (level_pad is
      // a multiple of F, so whole groups exist)
      if (wp < m) {
        float lo[D], hi[D];
#pragma unroll
        for (int d = 0; d < D; ++d) {
          lo[d] = __ldg(lmbr + d * lpad + l0 + lane);
          hi[d] = __ldg(lmbr + (D + d) * lpad + l0 + lane);
        }
        uint32_t any = 0;
        for (uint32_t j = wp; j < m; j += kJoinWarps) {
          BoxRow<D> b;
          b.load(bx + j * 2 * D);
          bool ov = lane < nl;
#pragma unroll
          for (int d = 0; d < D; ++d) ov &= overlaps1(-b.v[2 * d], b.v[2 * d + 1], lo[d], hi[d]);
          const uint32_t mov = __ballot_sync(0xffffffffu, ov);
          uint32_t mcov = 0, h = 0;
          if (mov) {  // warp-uniform
            bool in = ov;
#pragma unroll
            for (int d = 0; d < D; ++d) in &= inside1(-b.v[2 * d], b.v[2 * d + 1], lo[d], hi[d]);
            mcov = __ballot_sync(0xffffffffu, in);
            if (RECT && mcov && __ldg(t.inverted)) mcov = 0;
            if (mcov) {
              h = __popc(mcov) * F;
              // the tree's last leaf may hold fewer than F objects
              const uint64_t last = nleaves - 1 - l0;
              if (last < 32 && ((mcov >> last) & 1u)) h -= (uint32_t)(nleaves * F - t.n);
            }
          }
          any |= mov & ~mcov;
          if (lane == 0) {
            part[j] = mov & ~mcov;
            cov[j] = mcov;
            hits[j] = h;
          }
        }
        if (lane == 0 && any) atomicOr(&s_any, any);
      }
      __syncthreads();
      // room for the items' hit bits (one atomic) and where each one's start
      const uint32_t any = s_any;
      uint32_t off = kNoMask;
      if (hc.mask && any) {  // CTA-uniform
        const uint32_t words = tid < m ? __popc(part[tid]) * wpl : 0u;
        uint32_t wtot;
        const uint32_t ex = warp_excl_sum(words, &wtot);
        if (lane == 0) s_wsum[wp] = wtot;
        __syncthreads();
        uint32_t before = 0, total = 0;
#pragma unroll
        for (uint32_t w = 0; w < kJoinWarps; ++w) {
          const uint32_t c = s_wsum[w];
          before += w < wp ? c : 0u;
          total += c;
        }
        if (tid == 0) s_base = atomicAdd(hc.cursor, (unsigned long long)total);
        __syncthreads();
        if (words && s_base + total <= hc.mask_cap) off = (uint32_t)s_base + before + ex;
      }
      if (tid < m) moff[tid] = off;
      __syncthreads();
      // B. partially covered leaves: a warp per leaf, against every box that
      // overlaps it
      uint32_t held = 0;  // pairs whose hit bits are held
      auto flush = [&]() {
        __syncwarp();
        // eight bytes per lane, four lanes per pair
        const bool mine = lane / 4 < held;
        const uint32_t pr = mine ? pairs[lane / 4] : 0u;
        const uint2 w = mine ? reinterpret_cast<const uint2*>(bytes)[lane] : make_uint2(0, 0);
        const uint32_t j = pr & 0xffffu, k = (pr >> 16) & 0xffu, x = pr >> 24;
        uint32_t cnt = __popc(w.x) + __popc(w.y);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, 1);
        cnt += __shfl_xor_sync(0xffffffffu, cnt, 2);
        if (mine) {
          if ((lane & 3) == 0 && cnt) atomicAdd(&hits[j], cnt);
          const uint32_t at = moff[j];
          // by the leaf's place among the item's partially covered ones
          if (at != kNoMask)
            *reinterpret_cast<uint2*>(hc.mask + at + __popc(part[j] & ((1u << k) - 1u)) * wpl + x * kChunkWords +
                                      (lane & 3) * 2) = w;
        }
        held = 0;
        __syncwarp();
      };
      for (uint32_t k = wp; k < 32; k += kJoinWarps) {
        if (!((any >> k) & 1u)) continue;  // warp-uniform
        uint32_t np = 0;                   // pairs of this leaf
        for (uint32_t j0 = 0; j0 < m; j0 += 32) {
          const bool on = j0 + lane < m && ((part[j0 + lane] >> k) & 1u);
          const uint32_t sel = __ballot_sync(0xffffffffu, on);
          if (on) list[np + __popc(sel & lane_lt_mask())] = (uint16_t)(j0 + lane);
          np += __popc(sel);
        }
        __syncwarp();
        const uint64_t e0 = (l0 + k) * F;
        for (uint32_t x = 0; x < chunks; ++x) {
          const uint32_t o = x * 128 + lane * 4;
          Quad<D, RECT> c;
          if (o < F) load_quad<D, RECT>(c, t.coords, t.npad, e0 + o);
          // lanes past the leaf's end, objects past n (padding of the last leaf)
          uint32_t live = 0xfu;
          if (o >= F || e0 + o >= t.n) live = 0;
          else if (e0 + o + 4 > t.n) live = (1u << (t.n - e0 - o)) - 1u;
          for (uint32_t i = 0; i < np; ++i) {
            const uint32_t j = list[i];
            BoxRow<D> b;
            b.load(bx + j * 2 * D);
            uint32_t s[4] = {0, 0, 0, 0};
#pragma unroll
            for (int d = 0; d < D; ++d) miss_dim<D, RECT>(c, d, b.v[2 * d], b.v[2 * d + 1], s);
            bytes[held * 32 + lane] = (uint8_t)(hit_bits(s) & live);
            if (lane == 0) pairs[held] = j | (k << 16) | (x << 24);
            if (++held == kPairs) flush();
          }
        }
        __syncwarp();
      }
      if (held) flush();
      __syncthreads();
      if (tid < m) {
        const uint32_t cm = cov[tid], pm = part[tid], h = hits[tid];
        if (hc.rec) hc.rec[(i0 + a + tid) * G + g] = make_uint4(pm | cm, cm, moff[tid], h);
        if (h) atomicAdd(qcount + item[a + tid].x, (unsigned long long)h);
        if (stats) {
          n_cov += __popc(cm);
          n_part += __popc(pm);
          o_cov += __popc(cm) * F;
          const uint64_t last = nleaves - 1 - l0;
          if (last < 32 && ((cm >> last) & 1u)) o_cov -= nleaves * F - t.n;
        }
      }
      a += m;
      __syncthreads();  // the masks and boxes are free for the next node
    }
    if (tid == 0) s_task = fetched;
  }
  if (stats) {
    if (n_cov) atomicAdd(stats + kStatCovered, (unsigned long long)n_cov);
    if (n_part) atomicAdd(stats + kStatPartial, (unsigned long long)n_part);
    if (o_cov) atomicAdd(stats + kStatObjCovered, o_cov);
  }
}

// Leaves that an item overlaps and those that it covers partially, from one
// 32-leaf group each of eight items, a warp of the CTA each (every CTA takes the
// same ones, so all agree).  All threads call it.  With 32 groups the CTAs, which
// all pay for it, took 4 us of a call in 3-D and 12 in 8-D; with eight, 1 to 2.
struct Leaves {
  float overlapped, partial;
};
constexpr uint32_t kSampled = 8;
template <int D>
__device__ __forceinline__ Leaves leaves_per_item(const TreeView& t, const float* boxes, const uint2* items,
                                                  uint32_t nitems) {
  __shared__ uint32_t s_leaves[2];
  if (threadIdx.x < 2) s_leaves[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, G = t.fanout >> 5;
  const uint2 it = items[(uint64_t)w * nitems / kSampled];
  const uint64_t c = (uint64_t)it.y * t.fanout + w % G * 32 + lane;
  bool ov = false, in = false;
  if (c < t.nodes[0]) test_node<D>(load_box<D>(boxes, it.x), t.mbr[0], t.pad[0], c, ov, in);
  const uint32_t overlapped = __popc(__ballot_sync(0xffffffffu, ov));
  const uint32_t partial = __popc(__ballot_sync(0xffffffffu, ov && !in));
  if (lane == 0 && overlapped) {
    atomicAdd(&s_leaves[0], overlapped);
    atomicAdd(&s_leaves[1], partial);
  }
  __syncthreads();
  const float each = (float)G / kSampled;
  return {s_leaves[0] * each, s_leaves[1] * each};
}

// How the warps of k_count and k_leafwrite share the items: their 32-leaf groups
// in turn where those are fewer than four rounds of the grid's warps, up to eight
// unless an item has few leaves; from eight rounds on groups by need, each to the
// next free warp, where an item has many that it covers partially; whole items
// otherwise.
//   few leaves: 10,000 items of tiny boxes at fan-out 256, nine rounds: the
//   groups 66 us to count and 40 to write, whole items 44 and 23; a plan of 4,096
//   tiny boxes, two rounds of items: 201 and 164 us;
//   many covered ones: 1,500 8-D boxes of 75 leaves, five rounds: the groups 126
//   us to count, whole items 150;
//   many partially covered ones: whole items leave most warps waiting for the
//   last ones.  By need an atomic on one address per group is paid, about 1 ns
//   each: with 10 such leaves per item 9,000 boxes over 2 M points take 187 us by
//   items, 212 by need, with 22 6,000 over 1 M 233 and 217.
enum Share { kGroups, kItems, kGroupsByNeed };
static_assert(kSampled == 256 / 32, "a warp per sampled group");
constexpr float kManyPartial = 16.f, kFewLeaves = 8.f;
template <int D>
__device__ __forceinline__ Share share_items(const TreeView& t, const float* boxes, const uint2* items,
                                             uint32_t nitems, uint32_t G, uint32_t warps) {
  const uint64_t groups = (uint64_t)nitems * G;
  // (above four dimensions a box has leaves in many places and the sample reads
  // more: five rounds of 8-D groups 128 us to count, 138 with it)
  if (groups < (D > 4 ? 8ull : 4ull) * warps) return kGroups;
  if (groups >= 1u << 31) return kItems;  // (units are counted in 32 bits)
  const Leaves l = leaves_per_item<D>(t, boxes, items, nitems);
  if (groups < 8ull * warps) return l.overlapped < kFewLeaves ? kItems : kGroups;
  return l.partial >= kManyPartial ? kGroupsByNeed : kItems;
}

// Counts of batches that are not in node order: a warp per item or per 32-leaf
// group of one (share_items); no barriers.  Few items share a node, so nothing
// is staged: the box sits in registers, a group's MBRs are tested one per lane,
// and the partially covered leaves one after the other.  Bound by the latency
// of its dependent reads (item, box and MBRs, objects); more CTAs per SM hide it
// until the registers of a box, its MBRs and four objects spill too much
// (61,000 8-D points, 7,768 boxes: 110 -> 45 us with three instead of four;
// MBRs read one group ahead in one dimension only: 4 M 4-D rectangles 665 -> 626
// us without, 100,000 2-D points, 15,000 boxes 120 -> 111; 3-D points still spill
// 60 bytes, three CTAs were slower).  1,000 boxes
// over 1 M points: 18.9 (a warp per item) -> 12.4 us; 64 boxes over 16 M points
// 36.7 -> 14.8 us; 3,000 boxes with 34 leaves per item over 4 M 4-D rectangles
// at fan-out 256, by whole items in turn 900, by need 626.
template <int D, bool RECT>
__global__ void __launch_bounds__(256, (RECT ? 2 * D : D) > 8 ? 2 : (RECT ? 2 * D : D) > 3 ? 3 : 4)
    k_count(TreeView t, const float* __restrict__ boxes, const uint2* __restrict__ items,
            const uint32_t* __restrict__ item_count, uint32_t* work, unsigned long long* qcount, uint64_t item_cap,
            uint64_t nodes, unsigned long long* stats, HitCache hc) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t F = t.fanout, G = F >> 5;
  const uint32_t nitems = (uint32_t)min((uint64_t)*item_count, item_cap);
  if (is_ordered(nitems, nodes)) return;  // k_join's
  const uint64_t nleaves = t.nodes[0], lpad = t.pad[0];
  const float* lmbr = t.mbr[0];
  const uint32_t chunks = (F + 127u) >> 7, wpl = chunks * kChunkWords;
  const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
  // (points of seven and eight dimensions leave no registers for sharing by need:
  // with it 500,000 8-D points, 5,000 boxes take 167 us instead of 158)
  constexpr bool kMayNeed = RECT || D <= 6;
  Share share = (uint64_t)nitems * G < 8ull * warps ? kGroups : kItems;
  if constexpr (kMayNeed) share = share_items<D>(t, boxes, items, nitems, G, warps);
  const bool by_need = kMayNeed && share == kGroupsByNeed;
  const bool whole = share == kItems;
  const uint32_t units = whole ? nitems : nitems * G;
  // the next unit is known while this one is counted, so that its item is read
  // ahead: by need it has been asked for a unit earlier
  uint32_t asked = 0;  // lane 0's
  auto ask = [&]() {
    if (by_need && lane == 0) asked = atomicAdd(work, 1u);
  };
  auto after = [&](uint32_t u) {
    if (by_need) return __shfl_sync(0xffffffffu, asked, 0);
    return units - u > warps ? u + warps : units;
  };
  ask();
  uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (by_need) u = after(u);
  if (u >= units) return;
  ask();
  uint2 it = items[whole ? u : u / G];
  for (uint32_t un = after(u);;) {
    ask();
    uint2 next = it;
    if (un < units) next = items[whole ? un : un / G];
    float b[2 * D];  // -lo, hi per dimension, zeros as +0
    const float* q = boxes + (uint64_t)it.x * 2 * D;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const float lo = __ldg(q + d), hi = __ldg(q + D + d);
      b[2 * d] = lo == 0.f ? 0.f : -lo;
      b[2 * d + 1] = hi == 0.f ? 0.f : hi;
    }
    uint32_t total = 0;  // hits of the unit
    const uint32_t ga = whole ? 0u : u % G, gb = whole ? G : ga + 1;
    float mlo[D], mhi[D];  // a group's MBRs, in one dimension loaded one group ahead
    constexpr bool kMbrAhead = D == 1;
    auto load_mbrs = [&](uint32_t g) {
      const uint64_t at = (uint64_t)it.y * F + g * 32 + lane;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        mlo[d] = __ldg(lmbr + d * lpad + at);
        mhi[d] = __ldg(lmbr + (D + d) * lpad + at);
      }
    };
    if (kMbrAhead) load_mbrs(ga);
    for (uint32_t g = ga; g < gb; ++g) {
      if (!kMbrAhead) load_mbrs(g);
      const uint64_t l0 = (uint64_t)it.y * F + g * 32;  // the group's first leaf
      bool ov = l0 + lane < nleaves, in = true;
#pragma unroll
      for (int d = 0; d < D; ++d) {
        ov &= overlaps1(-b[2 * d], b[2 * d + 1], mlo[d], mhi[d]);
        in &= inside1(-b[2 * d], b[2 * d + 1], mlo[d], mhi[d]);
      }
      if (kMbrAhead && g + 1 < gb) load_mbrs(g + 1);
      const uint32_t mov = __ballot_sync(0xffffffffu, ov);
      uint32_t mcov = __ballot_sync(0xffffffffu, ov && in);
      if (RECT && mcov && __ldg(t.inverted)) mcov = 0;
      const uint32_t part = mov & ~mcov;
      // room for the hit bits; the objects' reads do not wait for it
      uint32_t off = kNoMask;
      const uint32_t words = __popc(part) * wpl;
      unsigned long long base = 0;
      if (hc.mask && words && lane == 0) base = atomicAdd(hc.cursor, (unsigned long long)words);
      uint32_t hits = 0;  // of this lane
      // the partially covered leaves' 128-object chunks, kAhead at a time
      constexpr uint32_t kAhead = (RECT ? 2 * D : D) <= 4 ? 2 : 1;
      const uint32_t nchunk = __popc(part) * chunks;
      uint32_t mp = part, x = 0;
      for (uint32_t c0 = 0; c0 < nchunk; c0 += kAhead) {
        Quad<D, RECT> c[kAhead];
        uint64_t p[kAhead];  // first object of the lane's four, t.n: none
#pragma unroll
        for (uint32_t v = 0; v < kAhead; ++v) {
          p[v] = t.n;
          if (c0 + v >= nchunk) continue;  // warp-uniform
          const uint32_t o = x * 128 + lane * 4;
          if (o < F) {
            p[v] = (l0 + __ffs(mp) - 1) * F + o;
            load_quad<D, RECT>(c[v], t.coords, t.npad, p[v]);
          }
          if (++x == chunks) {
            x = 0;
            mp &= mp - 1;
          }
        }
        if (hc.mask && c0 == 0) {
          base = __shfl_sync(0xffffffffu, base, 0);
          if (base + words <= hc.mask_cap) off = (uint32_t)base;
        }
#pragma unroll
        for (uint32_t v = 0; v < kAhead; ++v) {
          if (c0 + v >= nchunk) continue;
          uint32_t s[4] = {0, 0, 0, 0};
#pragma unroll
          for (int d = 0; d < D; ++d) miss_dim<D, RECT>(c[v], d, b[2 * d], b[2 * d + 1], s);
          uint32_t hm = hit_bits(s);
          // objects past n (padding of the last leaf) never hit
          if (p[v] + 4 > t.n) hm &= p[v] < t.n ? (1u << (t.n - p[v])) - 1u : 0u;
          hits += __popc(hm);
          if (off != kNoMask)
            reinterpret_cast<uint8_t*>(hc.mask + off + (c0 + v) * kChunkWords)[lane] = (uint8_t)hm;
        }
      }
      hits = __reduce_add_sync(0xffffffffu, hits);
      uint32_t chits = __popc(mcov) * F;
      // the tree's last leaf may hold fewer than F objects
      const uint64_t last = nleaves - 1 - l0;
      if (last < 32 && ((mcov >> last) & 1u)) chits -= (uint32_t)(nleaves * F - t.n);
      hits += chits;
      if (lane == 0) {
        if (hc.rec) hc.rec[whole ? (size_t)u * G + g : u] = make_uint4(mov, mcov, off, hits);
        if (stats) {
          if (mcov) atomicAdd(stats + kStatCovered, (unsigned long long)__popc(mcov));
          if (part) atomicAdd(stats + kStatPartial, (unsigned long long)__popc(part));
          if (chits) atomicAdd(stats + kStatObjCovered, (unsigned long long)chits);
        }
      }
      total += hits;
    }
    if (lane == 0 && total) atomicAdd(qcount + it.x, (unsigned long long)total);
    if (un >= units) break;
    u = un;
    un = after(u);
    it = next;
  }
}

// A warp per (query, level-1 node) item, or per 32-leaf group of one where the
// batch has too few items to keep the warps busy (64 boxes over 16 M points:
// 72 -> 22 us, the chain of one warp copying an item's up to 16,384 ids):
// the group's slot in the query's slice is reserved by its hit count, ids of
// covered leaves are copied as whole runs, ids of partially covered ones by
// their hit bits.  Bound by the writes of the ids and the latency in front of
// them: the records and slots of an item's groups are taken at once (one
// lane each), the hit bits of a group's leaves by one load, and four leaves'
// ids are in flight together.  qwhist: per-(query, window) id counts for the
// sort, gathered in per-warp shared counters and flushed once per fetch.
constexpr uint32_t kWriteUnroll = 4;
template <int D, bool RECT>
__global__ void __launch_bounds__(256) k_leafwrite(TreeView t, const float* __restrict__ boxes,
                                                   const uint2* __restrict__ items,
                                                   const uint32_t* __restrict__ item_count, uint32_t* work,
                                                   const uint4* __restrict__ rec, const uint32_t* __restrict__ hmask,
                                                   const unsigned long long* __restrict__ mask_words,
                                                   const unsigned long long* __restrict__ total_ids,
                                                   const unsigned long long* __restrict__ offsets,
                                                   unsigned long long* qcursor, int32_t* __restrict__ out,
                                                   uint64_t item_cap, uint32_t* qwhist, uint32_t hist_G,
                                                   uint32_t hist_bits) {
  __shared__ uint32_t wcount[8][kHistMaxG];
  const uint32_t lane = threadIdx.x & 31, lt = lane_lt_mask();
  uint32_t* wc = wcount[(threadIdx.x >> 5) & 7];
  const bool hist = qwhist != nullptr;
  if (hist) {
    for (uint32_t w = lane; w < hist_G; w += 32) wc[w] = 0;
    __syncwarp();
  }
  const uint32_t F = t.fanout, G = F >> 5;
  const uint32_t cpl = (F + 127u) >> 7;  // 128-object chunks per leaf
  const uint32_t nitems = (uint32_t)min((uint64_t)*item_count, item_cap);
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  // groups per fetch: a whole item, or one group in small batches; each warp's
  // first one by its index, more as the warps get free (all in turn, without
  // the atomic: 59 -> 87 us on the 15,000 items, a heavy item's groups follow
  // one another; all by the atomic: 13 -> 18 us for 1,000 boxes over 1 M points)
  // (from eight items per warp on whole ones leave no warp waiting for long: 16 M
  // points, 10,000 boxes of 10^9 ids 1.1 ms, by need 1.2)
  bool whole = nitems >= 8 * warps;
  if (!whole) {
    // the rule of share_items, without its sample where the count pass has
    // recorded hit bits: it asked for cpl * kChunkWords words per partially
    // covered leaf, and the ids make up F per covered one at least (the sample
    // comes out differently from call to call: 1.1 M points, 3,000 boxes, 19
    // partially covered leaves per item, 115 us one time and 170 the next)
    const uint64_t groups = (uint64_t)nitems * G;
    if (!hmask || groups < 4ull * warps) {
      whole = share_items<D>(t, boxes, items, nitems, G, warps) == kItems;
    } else {
      const float partial = (float)*mask_words / (float)(cpl * kChunkWords);
      whole = groups < 8ull * warps ? D <= 4 && partial + (float)*total_ids / (float)F < kFewLeaves * nitems
                                    : partial < kManyPartial * nitems;
    }
  }
  const uint32_t per = whole ? G : 1u;
  const uint32_t nfetch = whole ? nitems : nitems * G;
  for (uint32_t turn = 0;; ++turn) {
    uint32_t f = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (turn) {
      if (nfetch <= warps) break;
      if (lane == 0) f = warps + atomicAdd(work, 1u);
      f = __shfl_sync(0xffffffffu, f, 0);
    }
    if (f >= nfetch) break;
    const uint32_t i = whole ? f : f / G, gbase = whole ? 0u : f % G;
    const uint2 it = items[i];
    uint4 r = make_uint4(0, 0, kNoMask, 0);
    unsigned long long at = 0;
    if (lane < per) {
      r = rec[(size_t)i * G + gbase + lane];
      if (r.w) at = offsets[it.x] + atomicAdd(qcursor + it.x, (unsigned long long)r.w);
    }
    uint32_t todo = __ballot_sync(0xffffffffu, r.w != 0);
    if (!todo) continue;
    do {
      const uint32_t sl = __ffs(todo) - 1;
      todo &= todo - 1;
      const uint32_t mov = __shfl_sync(0xffffffffu, r.x, sl), mcov = __shfl_sync(0xffffffffu, r.y, sl);
      const uint32_t moff = __shfl_sync(0xffffffffu, r.z, sl);
      uint64_t wpos = __shfl_sync(0xffffffffu, at, sl);
      const uint64_t lb = (uint64_t)it.y * F + (gbase + sl) * 32;  // the group's first leaf
      uint32_t m = mcov;
      while (m) {
        // a run of consecutive covered leaves is one contiguous id range
        const int s = __ffs(m) - 1;
        const uint32_t shifted = ~(m >> s);
        const int len = shifted ? (__ffs(shifted) - 1) : (32 - s);
        m &= ~((len >= 32 ? 0xffffffffu : ((1u << len) - 1u)) << s);
        const uint64_t e0 = (lb + s) * F;
        uint64_t e1 = (lb + s + len) * F;
        if (e1 > t.n) e1 = t.n;
        const int32_t* src = t.ids + e0;
        const uint32_t cnt = (uint32_t)(e1 - e0);
        int32_t* dst = out + wpos;
        // eight loads in flight per lane before their stores
        uint32_t j = lane;
        for (; j + 224 < cnt; j += 256) {
          int32_t v[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) v[k] = __ldg(src + j + 32 * k);
#pragma unroll
          for (int k = 0; k < 8; ++k) dst[j + 32 * k] = v[k];
          if (hist) {
#pragma unroll
            for (int k = 0; k < 8; ++k) atomicAdd(wc + ((uint32_t)v[k] >> hist_bits), 1u);
          }
        }
        for (; j + 96 < cnt; j += 128) {
          int32_t v[4];
#pragma unroll
          for (int k = 0; k < 4; ++k) v[k] = __ldg(src + j + 32 * k);
#pragma unroll
          for (int k = 0; k < 4; ++k) dst[j + 32 * k] = v[k];
          if (hist) {
#pragma unroll
            for (int k = 0; k < 4; ++k) atomicAdd(wc + ((uint32_t)v[k] >> hist_bits), 1u);
          }
        }
        for (; j < cnt; j += 32) {
          const int32_t a = __ldg(src + j);
          dst[j] = a;
          if (hist) atomicAdd(wc + ((uint32_t)a >> hist_bits), 1u);
        }
        wpos += cnt;
      }
      // partially covered leaves: chunk c of the group's list is 128 objects
      // of its (c / cpl)-th leaf; its hit bits are the bytes of the words at
      // moff + kChunkWords c, or are found by testing the objects
      uint32_t mp = mov & ~mcov;
      const uint32_t nchunk = __popc(mp) * cpl;
      const bool cached = moff != kNoMask;
      uint32_t sub = 0;  // chunk of the leaf at mp's lowest bit
      const uint8_t* hb = reinterpret_cast<const uint8_t*>(hmask + moff) + lane;
      for (uint32_t c0 = 0; c0 < nchunk; c0 += kWriteUnroll) {
        uint32_t hm[kWriteUnroll];
        int4 idv[kWriteUnroll];
        if (cached) {
#pragma unroll
          for (uint32_t u = 0; u < kWriteUnroll; ++u)
            hm[u] = c0 + u < nchunk ? __ldg(hb + (c0 + u) * (kChunkWords * 4)) : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < kWriteUnroll; ++u) {
          idv[u] = make_int4(0, 0, 0, 0);
          if (!cached) hm[u] = 0;
          if (c0 + u >= nchunk) continue;  // warp-uniform
          const uint32_t o = sub * 128 + lane * 4;
          const uint64_t p = (lb + (__ffs(mp) - 1)) * F + o;
          if (++sub == cpl) {
            sub = 0;
            mp &= mp - 1;
          }
          if (!cached && o < F)
            hm[u] = test4_rolled<D, RECT>(boxes + (uint64_t)it.x * (2 * D), t.coords, t.npad, p, t.n);
          if (hm[u]) idv[u] = __ldg(reinterpret_cast<const int4*>(t.ids + p));
        }
#pragma unroll
        for (uint32_t u = 0; u < kWriteUnroll; ++u) {
          const int32_t ids[4] = {idv[u].x, idv[u].y, idv[u].z, idv[u].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const bool on = (hm[u] >> k) & 1u;
            const uint32_t w = __ballot_sync(0xffffffffu, on);
            if (on) {
              out[wpos + __popc(w & lt)] = ids[k];
              if (hist) atomicAdd(wc + ((uint32_t)ids[k] >> hist_bits), 1u);
            }
            wpos += __popc(w);
          }
        }
      }
    } while (todo);
    if (hist) {
      __syncwarp();
      for (uint32_t w = lane; w < hist_G; w += 32) {
        const uint32_t c = wc[w];
        if (c) {
          atomicAdd(qwhist + (size_t)it.x * hist_G + w, c);
          wc[w] = 0;
        }
      }
      __syncwarp();
    }
  }
}

// ---------------------------------------------------------------------------
// Plain traversal: one query per CTA, depth first, ids in key order.
//
// The CTA tests a node's children at once (one thread each) and keeps the
// level's overlap mask in shared memory; the overlapping leaves of successive
// level-1 nodes collect in a list of up to kPlainLeaves, which the warps then
// scan one leaf each.  Bound by the chain of the query with the most leaves:
// the list takes the barriers out of it (they were three per leaf, with one
// leaf in flight per CTA and a restart from the root after each run of hits:
// counting 1,000 boxes over 2 M points 197 -> 44 us, writing 291 -> 71).
// The write pass keeps a leaf's hit bits in shared memory while the list's
// counts are scanned into places.
// ---------------------------------------------------------------------------
constexpr uint32_t kPlainThreads = 256;
constexpr uint32_t kPlainWarps = kPlainThreads / 32;
constexpr uint32_t kPlainLeaves = 256;  // a node's children at most: one append always fits
static_assert(kPlainLeaves == kPlainThreads && kPlainLeaves >= kMaxFanout, "a thread per child and per listed leaf");

template <bool WRITE>
struct PlainSmem {
  uint32_t mask[kMaxLevels][kPlainWarps];  // overlapping children of the path's node at a level
  uint32_t list[kPlainLeaves];             // leaves, kPlainCovered if all of its objects are hits
  uint32_t sum[kPlainWarps];
  uint32_t cnt[WRITE ? kPlainLeaves : 1];
  uint8_t bits[WRITE ? kPlainLeaves : 1][WRITE ? kMaxFanout / 4 : 1];  // hit bits of four objects
};
constexpr uint32_t kPlainCovered = 0x80000000u;  // (leaves are below 2^31 / 32)

template <int D, bool RECT, int MODE>
__global__ void __launch_bounds__(kPlainThreads) k_mprs(TreeView t, const float* __restrict__ boxes, uint32_t nq,
                                                        unsigned long long* __restrict__ counts,
                                                        const unsigned long long* __restrict__ offsets,
                                                        int32_t* __restrict__ out) {
  constexpr bool kWr = MODE == kWrite;
  __shared__ PlainSmem<kWr> sm;
  const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5, lt = lane_lt_mask();
  const uint32_t F = t.fanout, top = t.levels - 1;

  for (uint32_t q = blockIdx.x; q < nq; q += gridDim.x) {
    const float* qb = boxes + (uint64_t)q * (2 * D);
    uint32_t hits = 0;  // this lane's share (count)
    uint64_t at = kWr ? offsets[q] : 0;
    uint32_t nlist = 0;

    // the listed leaves: one warp each; all threads call it
    auto scan_list = [&]() {
      __syncthreads();
      for (uint32_t e = w; e < nlist; e += kPlainWarps) {
        const uint32_t v = sm.list[e];
        const uint64_t e0 = (uint64_t)(v & ~kPlainCovered) * F;
        const uint32_t size = (uint32_t)min((uint64_t)F, t.n - e0);
        uint32_t c = 0;
        if (v & kPlainCovered) {
          if (lane == 0) c = size;
        } else {
          for (uint32_t o = lane * 4; o < F; o += 128) {
            const uint32_t m = test4_rolled<D, RECT>(qb, t.coords, t.npad, e0 + o, t.n);
            if (kWr) sm.bits[e][o >> 2] = (uint8_t)m;
            c += __popc(m);
          }
        }
        if (kWr) {
          c = __reduce_add_sync(0xffffffffu, c);
          if (lane == 0) sm.cnt[e] = c;
        } else {
          hits += c;
        }
      }
      __syncthreads();
      if (!kWr) return;
      // counts -> places within the list's ids
      const uint32_t mine = tid < nlist ? sm.cnt[tid] : 0;
      uint32_t inc = mine;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= (uint32_t)d) inc += y;
      }
      if (lane == 31) sm.sum[w] = inc;
      __syncthreads();
      uint32_t before = 0, total = 0;
#pragma unroll
      for (uint32_t k = 0; k < kPlainWarps; ++k) {
        const uint32_t x = sm.sum[k];
        if (k < w) before += x;
        total += x;
      }
      if (tid < nlist) sm.cnt[tid] = before + inc - mine;
      __syncthreads();
      for (uint32_t e = w; e < nlist; e += kPlainWarps) {
        const uint32_t v = sm.list[e];
        const uint64_t e0 = (uint64_t)(v & ~kPlainCovered) * F;
        const uint32_t size = (uint32_t)min((uint64_t)F, t.n - e0);
        int32_t* dst = out + at + sm.cnt[e];
        if (v & kPlainCovered) {
          for (uint32_t o = lane; o < size; o += 32) dst[o] = __ldg(t.ids + e0 + o);
        } else {
          for (uint32_t c = 0; c < F; c += 128) {
            const uint32_t o = c + lane * 4;
            const uint32_t m = o < F ? sm.bits[e][o >> 2] : 0u;
            int4 id = make_int4(0, 0, 0, 0);
            if (m) id = __ldg(reinterpret_cast<const int4*>(t.ids + e0 + o));
            const uint32_t b0 = __ballot_sync(0xffffffffu, m & 1u), b1 = __ballot_sync(0xffffffffu, m & 2u);
            const uint32_t b2 = __ballot_sync(0xffffffffu, m & 4u), b3 = __ballot_sync(0xffffffffu, m & 8u);
            int32_t* d = dst + __popc(b0 & lt) + __popc(b1 & lt) + __popc(b2 & lt) + __popc(b3 & lt);
            if (m & 1u) *d++ = id.x;
            if (m & 2u) *d++ = id.y;
            if (m & 4u) *d++ = id.z;
            if (m & 8u) *d = id.w;
            dst += __popc(b0) + __popc(b1) + __popc(b2) + __popc(b3);
          }
        }
      }
      at += total;
      __syncthreads();
    };

    if (top == 0) {
      if (tid == 0) sm.list[0] = 0;
      nlist = 1;
    } else {
      const Box<D> b = load_box<D>(boxes, q);
      uint32_t level = top;
      uint64_t node = 0;
      bool fresh = true;      // the node's children are not tested yet
      uint32_t next = 0;      // first child to look at
      for (;;) {
        if (fresh) {
          const uint64_t c = node * F + tid;
          bool ov = false, in = false;
          if (tid < F && c < t.nodes[level - 1]) test_node<D>(b, t.mbr[level - 1], t.pad[level - 1], c, ov, in);
          const uint32_t m = __ballot_sync(0xffffffffu, ov);
          __syncthreads();  // the masks' last use
          if (lane == 0) sm.mask[level][w] = m;
          __syncthreads();
          fresh = false;
          next = 0;
          if (level == 1) {
            uint32_t before = 0, total = 0;
#pragma unroll
            for (uint32_t k = 0; k < kPlainWarps; ++k) {
              const uint32_t x = __popc(sm.mask[1][k]);
              if (k < w) before += x;
              total += x;
            }
            if (nlist + total > kPlainLeaves) {
              scan_list();
              nlist = 0;
            }
            // (an object of a rectangle with lo > hi can miss a box that covers its leaf)
            if (ov) sm.list[nlist + before + __popc(m & lt)] = (uint32_t)c | (!RECT && in ? kPlainCovered : 0u);
            nlist += total;
            next = F;
          }
        }
        // the first overlapping child from `next` on
        uint32_t child = kPlainThreads;
        for (uint32_t k = next >> 5; k < kPlainWarps && next < F; ++k) {
          uint32_t m = sm.mask[level][k];
          if (k == next >> 5) m &= 0xffffffffu << (next & 31);
          if (m) {
            child = k * 32 + __ffs(m) - 1;
            break;
          }
        }
        if (child < F) {
          node = node * F + child;
          --level;
          fresh = true;
        } else if (level == top) {
          break;
        } else {
          next = (uint32_t)(node % F) + 1;
          node /= F;
          ++level;
        }
      }
    }
    if (nlist) scan_list();
    if (!kWr) {
      hits = __reduce_add_sync(0xffffffffu, hits);
      if (lane == 0) sm.sum[w] = hits;
      __syncthreads();
      if (tid == 0) {
        unsigned long long total = 0;
#pragma unroll
        for (uint32_t k = 0; k < kPlainWarps; ++k) total += sm.sum[k];
        counts[q] = total;
      }
    }
    __syncthreads();
  }
}

// in == nullptr: the root level of nroot queries.
template <int D>
void launch_expand(uint32_t grid, cudaStream_t s, const float* boxes, const uint2* in,
                   const uint32_t* in_count, uint32_t nroot, uint2* out, uint32_t* out_count, uint64_t cap,
                   const float* child_mbr, uint64_t nchild, uint64_t child_pad, uint32_t fanout,
                   uint32_t* overflow, uint32_t* need, uint32_t lanes = 32) {
  if (lanes == 8)
    k_expand<D, 8><<<grid, 256, 0, s>>>(boxes, in, in_count, nroot, out, out_count, cap, child_mbr, nchild, child_pad,
                                        fanout, overflow, need);
  else if (lanes == 16)
    k_expand<D, 16><<<grid, 256, 0, s>>>(boxes, in, in_count, nroot, out, out_count, cap, child_mbr, nchild,
                                         child_pad, fanout, overflow, need);
  else
    k_expand<D, 32><<<grid, 256, 0, s>>>(boxes, in, in_count, nroot, out, out_count, cap, child_mbr, nchild,
                                         child_pad, fanout, overflow, need);
}

// The count pass.  nodes == 0: k_count; otherwise the level-1 nodes of a batch
// that order_items has been over: k_count and k_join, one of which finds the
// batch to be the other's.  At most blocks_per_sm CTAs of 256 threads per SM
// (k_join's have 128), and no more of k_join's than are resident (its run
// length follows from the grid).
template <int D>
qcp_status launch_count(bool rect, uint64_t nodes, uint32_t blocks_per_sm, cudaStream_t s, const TreeView& t,
                        const float* boxes, const uint2* items, const uint32_t* item_count, uint32_t* work,
                        uint64_t* qcount, uint64_t item_cap, unsigned long long* stats, HitCache hc) {
  auto* count = rect ? k_count<D, true> : k_count<D, false>;
  count<<<(uint32_t)num_sms() * blocks_per_sm, 256, 0, s>>>(t, boxes, items, item_count, work,
                                                            (unsigned long long*)qcount, item_cap, nodes, stats, hc);
  note_launch();
  QCP_TRY(check_launch("k_count"));
  if (!nodes) return QCP_OK;
  auto* join = rect ? k_join<D, true> : k_join<D, false>;
  int fit = 0;
  QCP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, join, kJoinThreads, 0));
  const uint32_t per_sm = fit < 1 ? 1u : ((uint32_t)fit < 2 * blocks_per_sm ? (uint32_t)fit : 2 * blocks_per_sm);
  join<<<(uint32_t)num_sms() * per_sm, kJoinThreads, 0, s>>>(t, boxes, items, item_count, work,
                                                             (unsigned long long*)qcount, item_cap, nodes, stats, hc);
  note_launch();
  return check_launch("k_join");
}

template <int D>
void launch_leafwrite(bool rect, uint32_t grid, cudaStream_t s, const TreeView& t, const float* boxes,
                      const uint2* items, const uint32_t* item_count, uint32_t* work, const HitCache& hc,
                      const uint32_t* total_ids, const uint64_t* offsets, uint64_t* qcursor, int32_t* out, uint64_t item_cap, uint32_t* qwhist,
                      uint32_t hist_G, uint32_t hist_bits) {
  auto* kern = rect ? k_leafwrite<D, true> : k_leafwrite<D, false>;
  kern<<<grid, 256, 0, s>>>(t, boxes, items, item_count, work, hc.rec, hc.mask, hc.cursor,
                            (const unsigned long long*)total_ids, (const unsigned long long*)offsets,
                            (unsigned long long*)qcursor, out, item_cap, qwhist, hist_G, hist_bits);
}

template <int D, int MODE>
void launch_mprs(bool rect, uint32_t grid, cudaStream_t s, const TreeView& t,
                 const float* boxes, uint32_t nq, uint64_t* counts, const uint64_t* offsets,
                 int32_t* out) {
  if (rect)
    k_mprs<D, true, MODE><<<grid, kPlainThreads, 0, s>>>(t, boxes, nq, (unsigned long long*)counts,
                                                   (const unsigned long long*)offsets, out);
  else
    k_mprs<D, false, MODE><<<grid, kPlainThreads, 0, s>>>(t, boxes, nq, (unsigned long long*)counts,
                                                    (const unsigned long long*)offsets, out);
}

}  // namespace

// Grows the workspace buffers a batch of q queries needs before its items
// are known (items and output grow on demand below).
qcp_status ws_reserve_queries(qcp_index* ix, Workspace* ws, uint32_t q);
qcp_status ws_reserve_items(qcp_index* ix, Workspace* ws, size_t items);
qcp_status ws_reserve_out(qcp_index* ix, Workspace* ws, size_t ids);

qcp_status init_items(Workspace* ws, uint32_t q, cudaStream_t s) {
  k_init_items<<<(q + 255) / 256, 256, 0, s>>>(ws->items[0], q, 0, ws->ctr + kCtrFrontier0);
  note_launch();
  return QCP_OK;
}

// Items of level l (the root's: nroot queries, when cur < 0) in items[cur] ->
// items of level l - 1 in items[nxt].
static qcp_status expand_level(qcp_index* ix, Workspace* ws, uint32_t l, int cur, int nxt, uint32_t nroot,
                               cudaStream_t s) {
  const TreeView t = view_of(ix);
  const uint32_t grid = (uint32_t)num_sms() * ws->blocks_per_sm;
  uint32_t* ctr = ws->ctr;
  QCP_DISPATCH_D(ix->dims, launch_expand<DD>(grid, s, ws->qboxes, cur < 0 ? nullptr : ws->items[cur],
                                             ctr + kCtrFrontier0 + (cur < 0 ? 0 : cur), nroot,
                                             ws->items[nxt], ctr + kCtrFrontier0 + nxt, ws->items_cap,
                                             t.mbr[l - 1], t.nodes[l - 1], t.pad[l - 1], t.fanout,
                                             ctr + kCtrOverflow, ctr + kCtrNeedItems, ws->lanes_per_item));
  note_launch();
  return check_launch("k_expand");
}

// Level-1 nodes of a batch whose items may be put in node order (four launches)
// and counted by k_join, 0 for one that is not: many queries, and more leaves
// than stay close to every warp anyway (the order alone is worth little:
// 1 M points, 7,813 leaves, 10,000 boxes 105 us with it, 102 without; 103,699
// rectangles, 2,502 boxes 39 and 15).  16 M points, 10,000 boxes: 306 us, 586
// without; 64 M 2-D points 262, 377; 32 M 8-D rectangles 0.85 ms, 3.4.
constexpr uint32_t kNodeOrderMinQueries = 1024;
constexpr uint64_t kNodeOrderMinLeaves = 16384;

static uint64_t order_nodes(const qcp_index* ix, uint32_t q) {
  const bool may = q >= kNodeOrderMinQueries && ix->levels > 2 && ix->level_nodes[0] >= kNodeOrderMinLeaves &&
                   q >= ix->level_nodes[1];
  return may ? ix->level_nodes[1] : 0;
}

// The level-1 items in items[*cur] in node order, into the other buffer.  hist:
// twice as many words as there are level-1 nodes; scan: scan_scratch_bytes of
// their number.
static qcp_status order_items(qcp_index* ix, uint2* const* items, size_t item_cap, uint32_t* ctr, uint32_t* hist,
                              void* scan, size_t scan_bytes, int* cur, cudaStream_t s) {
  const uint32_t grid = (uint32_t)num_sms() * 8;
  const int nxt = *cur ^ 1;
  const uint64_t nodes = ix->level_nodes[1];
  QCP_CUDA(cudaMemsetAsync(hist, 0, sizeof(uint32_t) * nodes, s));
  k_node_hist<<<grid, 256, 0, s>>>(items[*cur], ctr + kCtrFrontier0 + *cur, item_cap, nodes, hist);
  uint32_t* cursor = hist + nodes;
  QCP_TRY(exclusive_scan<uint32_t>(hist, cursor, nodes, nullptr, ix->pool, s, scan, scan_bytes));
  k_node_scatter<<<grid, 256, 0, s>>>(items[*cur], ctr + kCtrFrontier0 + *cur, item_cap, nodes, cursor, items[nxt],
                                      ctr + kCtrFrontier0 + nxt);
  note_launch(2);
  *cur = nxt;
  return check_launch("order_items");
}
static qcp_status order_items(qcp_index* ix, Workspace* ws, int* cur, cudaStream_t s) {
  return order_items(ix, ws->items, ws->items_cap, ws->ctr, ws->node_hist, ws->scan_tmp, ws->scan_tmp_cap, cur, s);
}

// What the count pass of this call records for its write pass.
static HitCache hit_cache_of(Workspace* ws) {
  const bool bits = ws->use_hit_cache && ws->hmask;
  return HitCache{ws->item_grp, bits ? ws->hmask : nullptr,
                  (uint32_t)(ws->hmask_cap > 0xfffffff0u ? 0xfffffff0u : ws->hmask_cap),
                  reinterpret_cast<unsigned long long*>(ws->ctr + kCtrMaskWords)};
}

static qcp_status count_items(qcp_index* ix, Workspace* ws, uint32_t q, int cur, bool counts_only, cudaStream_t s) {
  const TreeView t = view_of(ix);
  uint32_t* ctr = ws->ctr;
  const HitCache hc = counts_only ? HitCache{} : hit_cache_of(ws);
  qcp_status st = QCP_OK;
  QCP_DISPATCH_D(ix->dims, st = launch_count<DD>(ix->is_rect != 0, order_nodes(ix, q), ws->blocks_per_sm, s, t, ws->qboxes, ws->items[cur],
                                                ctr + kCtrFrontier0 + cur, ctr + kCtrWork, ws->qcount,
                                                ws->items_cap, ws->timing ? ws->d_stats : nullptr, hc));
  return st;
}

static qcp_status write_items(qcp_index* ix, Workspace* ws, int cur, cudaStream_t s) {
  const TreeView t = view_of(ix);
  const uint32_t grid = (uint32_t)num_sms() * ws->blocks_per_sm;
  uint32_t* ctr = ws->ctr;
  QCP_DISPATCH_D(ix->dims, launch_leafwrite<DD>(ix->is_rect != 0, grid, s, t, ws->qboxes, ws->items[cur],
                                                ctr + kCtrFrontier0 + cur, ctr + kCtrWrite, hit_cache_of(ws),
                                                ctr + kCtrTotal, ws->offsets, ws->qcursor, ws->out_ids, ws->items_cap,
                                                ws->hist_G ? ws->qwhist : nullptr, ws->hist_G, ws->hist_bits));
  note_launch();
  return check_launch("k_leafwrite");
}

// The call's counters to the host (and the total to h_total).
static qcp_status read_counters(Workspace* ws, cudaStream_t s) {
  QCP_CUDA(cudaMemcpyAsync(ws->h_ctr, ws->ctr, sizeof(uint32_t) * kCtrCount, cudaMemcpyDeviceToHost, s));
  QCP_CUDA(cudaStreamSynchronize(s));
  memcpy(ws->h_total, ws->h_ctr + kCtrTotal, sizeof(uint64_t));
  return QCP_OK;
}

// The bounded waits of the window sort's bulk prefetch.
static qcp_status check_timeout(Workspace* ws, cudaStream_t s) {
  QCP_CUDA(cudaMemcpyAsync(ws->h_ctr + kCtrTimeout, ws->ctr + kCtrTimeout, sizeof(uint32_t), cudaMemcpyDeviceToHost,
                           s));
  QCP_CUDA(cudaStreamSynchronize(s));
  if (ws->h_ctr[kCtrTimeout]) {
    set_error("a bounded wait for a bulk copy ran out in the sort");
    return QCP_ERR_TIMEOUT;
  }
  return QCP_OK;
}

qcp_status run_batched(qcp_index* ix, Workspace* ws, uint32_t q, bool counts_only, bool sort,
                       cudaStream_t s) {
  uint32_t* ctr = ws->ctr;
  // start level: items at level `start` are (query, node) pairs
  const uint32_t start = (ix->levels >= 2) ? ix->levels - 1 : 1;
  const bool order = order_nodes(ix, q) != 0;
  if (order) QCP_TRY(ws_reserve_nodes(ws, ix->level_nodes[1]));
  ws->use_hit_cache = false;
  for (int attempt = 0; attempt < 8; ++attempt) {
    mark(ws, kEvStart, s);
    QCP_CUDA(ws_zero(ws, q, s));
    if (ws->timing) QCP_CUDA(cudaMemsetAsync(ws->d_stats, 0, sizeof(unsigned long long) * kStatCount, s));
    // the GPU's first level: the root's, or the hand-off level of a CPU + GPU
    // co-processing call whose host threads walked the levels above
    uint32_t gpu_start = start;
    if (ws->hybrid) {
      gpu_start = ws->handoff_level < 1 ? 1u : (ws->handoff_level > start ? start : ws->handoff_level);
    }
    // frontier sizes of the levels (kStatLevel0 slots), for timed calls
    auto note_level = [&](uint32_t l, int slot) -> qcp_status {
      if (ws->timing)
        QCP_CUDA(cudaMemcpyAsync(ws->d_stats + kStatLevel0 + l, ctr + kCtrFrontier0 + slot, sizeof(uint32_t),
                                 cudaMemcpyDeviceToDevice, s));
      return QCP_OK;
    };
    int cur = 0;
    bool root = false;  // the next expansion starts from the root's implied items
    if (gpu_start < start) {
      QCP_TRY(host_frontier(ix, ws, q, gpu_start, s));
    } else if (gpu_start == 1 || ws->timing) {
      QCP_TRY(init_items(ws, q, s));
    } else {
      root = true;
    }
    if (!root) QCP_TRY(note_level(gpu_start, cur));
    const uint32_t held = root ? gpu_start - 1 : gpu_start;  // first level whose items are in a buffer
    for (uint32_t l = gpu_start; l > 1; --l) {
      const int nxt = root ? 0 : cur ^ 1;
      // (from then on the output counter is that of the items of two levels up)
      if (l < held) QCP_CUDA(cudaMemsetAsync(ctr + kCtrFrontier0 + nxt, 0, sizeof(uint32_t), s));
      QCP_TRY(expand_level(ix, ws, l, root ? -1 : cur, nxt, q, s));
      QCP_TRY(note_level(l - 1, nxt));
      cur = nxt;
      root = false;
    }
    if (order) QCP_TRY(order_items(ix, ws, &cur, s));
    mark(ws, kEvExpand, s);
    // a call that writes ids keeps the count pass's hits for the write pass
    ws->use_hit_cache = !counts_only && ws->hit_cache_on;
    if (!counts_only)
      QCP_TRY(ws_reserve_hitcache(ws, ws->items_cap * (ix->fanout / 32),
                                  ws->use_hit_cache && !ws->hmask_cap ? (size_t)1 << 21 : 0));
    QCP_TRY(count_items(ix, ws, q, cur, counts_only, s));
    mark(ws, kEvCount, s);
    if (!counts_only) {
      QCP_TRY(exclusive_scan_counts(ws->qcount, ws->offsets, q, ix->pool, s));
      QCP_TRY(classify_slices(ix, ws, q, sort, ~0ull, nullptr, s));
    }
    mark(ws, kEvScan, s);
    // one readback: overflow flags, items needed, total hits, job counts
    QCP_TRY(read_counters(ws, s));
    if (ws->h_ctr[kCtrOverflow]) {
      size_t need = (size_t)ws->h_ctr[kCtrNeedItems];
      if (need < ws->items_cap * 2) need = ws->items_cap * 2;
      QCP_TRY(ws_reserve_items(ix, ws, need));
      continue;
    }
    if (counts_only) return QCP_OK;
    const uint64_t total = *ws->h_total;
    QCP_TRY(ws_reserve_out(ix, ws, (size_t)total));
    if (total) {
      ws->hist_G = 0;
      const bool windows = sort && ws->h_ctr[kCtrJobs1];
      if (windows) {  // the write pass counts ids per (query, sort window)
        uint32_t wbits = 0, G = 0;
        sort_window_shape(ix, ws, &wbits, &G);
        if (G <= kHistMaxG) {
          QCP_TRY(ws_reserve_qwhist(ws, (size_t)q * G));
          QCP_CUDA(cudaMemsetAsync(ws->qwhist, 0, sizeof(uint32_t) * q * G, s));
          ws->hist_G = G;
          ws->hist_bits = wbits;
        }
      }
      QCP_TRY(write_items(ix, ws, cur, s));
      mark(ws, kEvWrite, s);
      if (sort) QCP_TRY(segmented_sort(ix, ws, s));
      mark(ws, kEvSort, s);
      if (windows) QCP_TRY(check_timeout(ws, s));
    }
    // hit bits that did not fit this call were tested again by the write
    // pass; the next call gets room for them (after this call's passes)
    if (ws->use_hit_cache) {
      uint64_t words;
      memcpy(&words, ws->h_ctr + kCtrMaskWords, sizeof(words));
      if (words > ws->hmask_cap && ws->hmask_cap < kMaxMaskWords) {
        QCP_CUDA(cudaStreamSynchronize(s));
        QCP_TRY(ws_reserve_hitcache(ws, 0, (size_t)(words < kMaxMaskWords ? words : kMaxMaskWords)));
      }
    }
    ws->use_hit_cache = false;
    return QCP_OK;
  }
  set_error("query frontier did not fit after repeated growth");
  return QCP_ERR_OOM;
}

qcp_status run_plain(qcp_index* ix, Workspace* ws, uint32_t q, bool counts_only, bool sort,
                     cudaStream_t s) {
  const TreeView t = view_of(ix);
  const uint32_t D = ix->dims;
  const bool rect = ix->is_rect != 0;
  uint32_t grid = q ? q : 1;
  if (grid > (uint32_t)num_sms() * 64) grid = (uint32_t)num_sms() * 64;
  mark(ws, kEvStart, s);
  QCP_CUDA(ws_zero(ws, 0, s));
  if (ws->timing) QCP_CUDA(cudaMemsetAsync(ws->d_stats, 0, sizeof(unsigned long long) * kStatCount, s));
  mark(ws, kEvExpand, s);
  QCP_DISPATCH_D(D, launch_mprs<DD, kCount>(rect, grid, s, t, ws->qboxes, q, ws->qcount,
                                            nullptr, nullptr));
  note_launch();
  QCP_TRY(check_launch("k_mprs<count>"));
  mark(ws, kEvCount, s);
  if (counts_only) {
    mark(ws, kEvScan, s);
    return QCP_OK;
  }
  QCP_TRY(exclusive_scan_counts(ws->qcount, ws->offsets, q, ix->pool, s));
  QCP_TRY(classify_slices(ix, ws, q, sort, ~0ull, nullptr, s));
  mark(ws, kEvScan, s);
  QCP_TRY(read_counters(ws, s));
  const uint64_t total = *ws->h_total;
  QCP_TRY(ws_reserve_out(ix, ws, (size_t)total));
  if (total) {
    ws->hist_G = 0;  // the sort counts its windows itself
    QCP_DISPATCH_D(D, launch_mprs<DD, kWrite>(rect, grid, s, t, ws->qboxes, q, nullptr,
                                              ws->offsets, ws->out_ids));
    note_launch();
    QCP_TRY(check_launch("k_mprs<write>"));
    mark(ws, kEvWrite, s);
    if (sort) QCP_TRY(segmented_sort(ix, ws, s));
    mark(ws, kEvSort, s);
    if (sort && ws->sort_msd_jobs) QCP_TRY(check_timeout(ws, s));
  }
  return QCP_OK;
}

// Batched per-query hit counts into caller-provided device buffers (boxes,
// counts) with scratch supplied by the caller as well: two frontier buffers
// of item_cap items, kCtrCount counters, and for up to max_nodes level-1 nodes
// what order_items needs (more are counted as they come).  Nothing is allocated.  Returns
// QCP_ERR_OUTPUT_OVERFLOW when the batch's frontier exceeds item_cap.
qcp_status run_batched_counts_into(qcp_index* ix, const float* boxes, uint32_t q, uint64_t* counts,
                                   uint2* items0, uint2* items1, size_t item_cap, uint32_t* ctr, uint32_t* hist,
                                   size_t max_nodes, void* scan, size_t scan_bytes, cudaStream_t s) {
  const TreeView t = view_of(ix);
  const uint32_t D = ix->dims;
  const bool rect = ix->is_rect != 0;
  const uint32_t grid = (uint32_t)num_sms() * 8;
  uint2* items[2] = {items0, items1};
  const uint32_t start = (ix->levels >= 2) ? ix->levels - 1 : 1;
  QCP_CUDA(cudaMemsetAsync(ctr, 0, sizeof(uint32_t) * kCtrCount, s));
  QCP_CUDA(cudaMemsetAsync(counts, 0, sizeof(uint64_t) * q, s));
  int cur = 0;
  if (start == 1) {
    k_init_items<<<(q + 255) / 256, 256, 0, s>>>(items[0], q, 0, ctr + kCtrFrontier0);
    note_launch();
  }
  for (uint32_t l = start; l > 1; --l) {
    const bool root = l == start;
    const int nxt = root ? 0 : cur ^ 1;
    if (l + 1 < start) QCP_CUDA(cudaMemsetAsync(ctr + kCtrFrontier0 + nxt, 0, sizeof(uint32_t), s));
    QCP_DISPATCH_D(D, launch_expand<DD>(grid, s, boxes, root ? nullptr : items[cur], ctr + kCtrFrontier0 + cur, q,
                                        items[nxt], ctr + kCtrFrontier0 + nxt, item_cap, t.mbr[l - 1], t.nodes[l - 1],
                                        t.pad[l - 1], t.fanout, ctr + kCtrOverflow, ctr + kCtrNeedItems));
    note_launch();
    cur = nxt;
  }
  uint64_t nodes = order_nodes(ix, q);
  if (nodes > max_nodes) nodes = 0;
  if (nodes) QCP_TRY(order_items(ix, items, item_cap, ctr, hist, scan, scan_bytes, &cur, s));
  qcp_status st = QCP_OK;
  QCP_DISPATCH_D(D, st = launch_count<DD>(rect, nodes, 8, s, t, boxes, items[cur], ctr + kCtrFrontier0 + cur,
                                         ctr + kCtrWork, counts, item_cap, nullptr, HitCache{}));
  QCP_TRY(st);
  uint32_t overflow = 0;  // pageable host word: no pinned buffer is allocated
  QCP_CUDA(cudaMemcpyAsync(&overflow, ctr + kCtrOverflow, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  QCP_CUDA(cudaStreamSynchronize(s));
  if (overflow) {
    set_error("query frontier exceeds the fixed scratch of this entry point; split the batch");
    return QCP_ERR_OUTPUT_OVERFLOW;
  }
  return QCP_OK;
}


// The batched pipeline with fixed capacities and no host readback: the
// frontier overflow (bit 1) and the id-capacity overflow (bit 2) are left in
// ws->ctr[kCtrOverflow] for the caller to read after the stream has run; on
// either, the results are incomplete.  All buffers must be reserved before
// (ws_reserve_*, ws->out_cap >= ids_cap); sort tables as segmented_sort_device.
// Stream-capturable.
qcp_status run_batched_device(qcp_index* ix, Workspace* ws, uint32_t q, uint64_t ids_cap, bool sort,
                              void* sort_tables, cudaStream_t s) {
  uint32_t* ctr = ws->ctr;
  const uint32_t start = (ix->levels >= 2) ? ix->levels - 1 : 1;
  ws->use_hit_cache = ws->hmask != nullptr;
  if (ws->hist_G) {  // needed by the write pass only: beside the traversal
    QCP_CUDA(ws_branch(ws, 0, s, ws->side));
    QCP_CUDA(cudaMemsetAsync(ws->qwhist, 0, sizeof(uint32_t) * q * ws->hist_G, ws->side));
  }
  QCP_CUDA(ws_zero(ws, q, s));
  int cur = 0;
  if (start == 1) QCP_TRY(init_items(ws, q, s));
  for (uint32_t l = start; l > 1; --l) {
    const bool root = l == start;
    const int nxt = root ? 0 : cur ^ 1;
    if (l + 1 < start) QCP_CUDA(cudaMemsetAsync(ctr + kCtrFrontier0 + nxt, 0, sizeof(uint32_t), s));
    QCP_TRY(expand_level(ix, ws, l, root ? -1 : cur, nxt, q, s));
    cur = nxt;
  }
  if (order_nodes(ix, q)) QCP_TRY(order_items(ix, ws, &cur, s));
  QCP_TRY(count_items(ix, ws, q, cur, false, s));
  QCP_TRY(exclusive_scan_counts(ws->qcount, ws->offsets, q, ix->pool, s, ws->scan_tmp, ws->scan_tmp_cap));
  // a batch of more than ids_cap ids: flagged, nothing written or sorted
  QCP_TRY(classify_slices(ix, ws, q, sort, ids_cap, ctr + kCtrFrontier0 + cur, s));
  if (ws->hist_G) QCP_CUDA(ws_branch(ws, 1, ws->side, s));
  QCP_TRY(write_items(ix, ws, cur, s));
  if (sort) QCP_TRY(segmented_sort_device(ix, ws, q, sort_tables, s));
  return check_launch("batched pipeline (device counts)");
}


// ---------------------------------------------------------------------------
// CPU + GPU co-processing: the host walks the internal levels.
//
// The reference's Hybrid::Search (src/tree/hybrid.cpp:451-760) gives every
// host thread a share of the queries; per query the thread walks the upper
// tree (Hybrid::TraverseInternalNodes, :801-960) to a run of leaf nodes and
// launches a GPU scan of that run, one launch per run.  Here the host threads
// walk every query of the batch down to the hand-off level at once and the
// GPU gets the whole frontier in one copy; expansion below the hand-off
// level, the leaf scan, the write and the sort stay on the GPU.  The host
// uses a copy of the internal levels' MBRs and the same closed-interval
// predicate as the kernels.
// ---------------------------------------------------------------------------
static qcp_status ensure_host_mbr(qcp_index* ix) {
  std::lock_guard<std::mutex> g(ix->host_mbr_mu);
  if (ix->host_mbr_ready) return QCP_OK;
  for (uint32_t l = 1; l < ix->levels; ++l) {
    const size_t n = 2 * (size_t)ix->dims * ix->level_pad[l];
    ix->host_mbr[l].resize(n);
    QCP_CUDA(cudaMemcpy(ix->host_mbr[l].data(), ix->mbr[l], sizeof(float) * n, cudaMemcpyDeviceToHost));
  }
  ix->host_mbr_ready = true;
  return QCP_OK;
}

qcp_status host_frontier(qcp_index* ix, Workspace* ws, uint32_t q, uint32_t level, cudaStream_t s) {
  QCP_TRY(ensure_host_mbr(ix));
  const uint32_t D = ix->dims, F = ix->fanout, top = ix->levels - 1;
  const float* boxes = ws->h_boxes;
  uint32_t T = ws->cpu_threads ? ws->cpu_threads : std::thread::hardware_concurrency();
  if (T == 0) T = 1;
  if (T > 64) T = 64;
  if (T > q) T = q ? q : 1;
  std::vector<std::vector<uint2>> part(T);
  auto walk = [&](uint32_t t) {
    const uint32_t q0 = (uint32_t)((uint64_t)q * t / T), q1 = (uint32_t)((uint64_t)q * (t + 1) / T);
    std::vector<std::pair<uint32_t, uint64_t>> stack;  // (level, node)
    auto& out = part[t];
    for (uint32_t qq = q0; qq < q1; ++qq) {
      const float* b = boxes + (size_t)qq * 2 * D;
      stack.clear();
      stack.emplace_back(top, 0);
      while (!stack.empty()) {
        const uint32_t l = stack.back().first;
        const uint64_t node = stack.back().second;
        stack.pop_back();
        const uint32_t cl = l - 1;
        const float* m = ix->host_mbr[cl].data();
        const uint64_t pad = ix->level_pad[cl];
        const uint64_t c0 = node * F;
        const uint64_t c1 = std::min<uint64_t>(c0 + F, ix->level_nodes[cl]);
        // children in reverse so that the stack pops them in order
        for (uint64_t c = c1; c-- > c0;) {
          bool ov = true;
          for (uint32_t d = 0; d < D && ov; ++d) ov = overlaps1(b[d], b[D + d], m[d * pad + c], m[(D + d) * pad + c]);
          if (!ov) continue;
          if (cl == level) out.push_back(make_uint2(qq, (uint32_t)c));
          else stack.emplace_back(cl, c);
        }
      }
    }
  };
  std::vector<std::thread> pool;
  for (uint32_t t = 1; t < T; ++t) pool.emplace_back(walk, t);
  walk(0);
  for (auto& th : pool) th.join();
  size_t n = 0;
  for (auto& p : part) n += p.size();
  ws->h_items.resize(n ? n : 1);
  size_t k = 0;
  for (auto& p : part) {
    std::copy(p.begin(), p.end(), ws->h_items.begin() + k);
    k += p.size();
  }
  if (n > 0xffffffffull) {
    set_error("co-processing frontier exceeds 2^32 items");
    return QCP_ERR_OOM;
  }
  QCP_TRY(ws_reserve_items(ix, ws, n));
  ws->h_nitems = (uint32_t)n;
  if (n) QCP_CUDA(cudaMemcpyAsync(ws->items[0], ws->h_items.data(), sizeof(uint2) * n, cudaMemcpyHostToDevice, s));
  QCP_CUDA(cudaMemcpyAsync(ws->ctr + kCtrFrontier0, &ws->h_nitems, sizeof(uint32_t), cudaMemcpyHostToDevice, s));
  // pageable sources: wait for the copies before the host vectors change
  QCP_CUDA(cudaStreamSynchronize(s));
  return QCP_OK;
}

}  // namespace qcp
