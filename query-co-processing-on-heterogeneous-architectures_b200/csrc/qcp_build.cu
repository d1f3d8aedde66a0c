// Device bulk load: Hilbert keys -> LSD radix sort of (key, id) -> packing
// into sorted SoA coordinate arrays -> bottom-up MBR levels.
//
// Replaces the host-threaded steps of the reference build
// (src/tree/tree.cpp:544-639 branch creation and key mapping,
// src/sort/thrust_sorter.cpp:12-47 sort and rank reassignment,
// src/tree/tree.cpp:683-745 packing, :410-495 and :1025-1133 bottom-up
// build, src/transformer/transformer.cpp:52-88 AoS->SoA transform): every
// step runs on the device and nothing crosses PCIe between them.
//
// Layout in HBM (see qcp_index):
//   coords[c * npad + i]   coordinate c of the i-th object in key order
//   ids[i]                 input id of the i-th object in key order
//   mbr[l][c * pad_l + k]  MBR component c ([lo0..lo(D-1), hi0..hi(D-1)]) of
//                          node k of level l (level 0 = leaves)
// Node k of level l covers children [k*F, (k+1)*F) of level l-1; leaf j
// covers objects [j*F, (j+1)*F).  No child pointers are stored.
#include <cfloat>
#include <cmath>

#include "qcp_internal.cuh"
#include "qcp_tree.cuh"

namespace qcp {

namespace {

__device__ __forceinline__ int64_t quantise(float p, uint32_t bits, uint32_t mode) {
  if (mode == QCP_KEY_REF) {
    // (long long)(1000000 * p): single-precision multiply then truncation
    // (src/mapper/hilbert_mapper.cpp:21-23)
    return (int64_t)__fmul_rn(1000000.0f, p);
  }
  float v = (p > 0.0f) ? p : 0.0f;  // negatives and NaN -> 0
  uint64_t maxq = low_ones64(bits);
  if (v >= 1.0f) return (int64_t)maxq;
  uint64_t q = (uint64_t)__fmul_rn(v, (float)(1ull << bits));  // exact scaling
  return (int64_t)(q > maxq ? maxq : q);
}

// quantise for QCP_KEY_NORM and bits <= 32, where every result fits 32 bits
// (a product of v < 1 stays below 2^bits): one 32-bit conversion.
__device__ __forceinline__ uint32_t quantise_norm32(float p, float scale, uint32_t maxq) {
  const float v = (p > 0.0f) ? p : 0.0f;  // negatives and NaN -> 0
  return v >= 1.0f ? maxq : __float2uint_rz(__fmul_rn(v, scale));
}

// One thread per object, the dimension count a template parameter so that the
// coordinates stay in registers; *max_key becomes the largest key.
//
// Normalised keys go through a table of HilbertTab<D>::L levels per lookup in
// shared memory, filled by every block from hilbert_step: the Gray code of the
// transposed bit levels is c ^ (c >> 1) of each coordinate, and the table is
// indexed by the coordinates' L-bit fields side by side, so no bit is ever
// interleaved.  Reference keys, whose coordinates may be wider than a field or
// negative, take the general form.  Bound by issue; before, the bits were
// interleaved first, and only 2-D and 3-D keys had a table: 16 M 3-D points
// 227 -> 190 us, 5 M 4-D rectangles 237 -> 86 us.
template <int D>
__global__ void __launch_bounds__(256) k_keys(const float* __restrict__ objs, uint64_t n, uint32_t is_rect,
                                              uint32_t mode, uint32_t bits, uint64_t* __restrict__ keys,
                                              unsigned long long* max_key) {
  constexpr uint32_t L = HilbertTab<D>::L, IB = L * D;
  extern __shared__ uint16_t tab[];
  if (mode == QCP_KEY_NORM && D > 1) {
    for (uint32_t e = threadIdx.x; e < hilbert_tab_size<D>(); e += blockDim.x) tab[e] = hilbert_field_entry<D>(e);
    __syncthreads();
  }
  const uint32_t stride = is_rect ? 2 * D : D;
  const float scale = (float)(1ull << bits);
  const uint32_t maxq = (uint32_t)low_ones64(bits);
  const uint64_t low_bits = bits > 1 ? dilate<D>(low_ones64(bits), bits) >> 1 : 0;  // as in hilbert_finish
  uint64_t most = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const float* o = objs + i * stride;
    float p[D];
#pragma unroll
    for (int d = 0; d < D; ++d)
      p[d] = is_rect ? __fmul_rn(0.5f, __fadd_rn(__ldg(o + d), __ldg(o + D + d))) : __ldg(o + d);
    uint64_t key;
    if (mode == QCP_KEY_NORM && D > 1) {
      uint32_t c[D];
#pragma unroll
      for (int d = 0; d < D; ++d) {
        const uint32_t q = quantise_norm32(p[d], scale, maxq);
        c[d] = bits > 1 ? q ^ (q >> 1) : q;  // a single level is not Gray-coded
      }
      key = 0;
      uint32_t state = 0;
      int lvl = (int)bits;  // levels left
      for (; lvl >= (int)L; lvl -= (int)L) {
        uint32_t in = 0;
#pragma unroll
        for (int d = 0; d < D; ++d) in |= ((c[d] >> (lvl - (int)L)) & ((1u << L) - 1u)) << (d * L);
        const uint32_t e = tab[(state << IB) | in];
        key = (key << IB) | (e & ((1u << IB) - 1u));
        state = e >> IB;
      }
      // bits % L levels
      uint32_t rot = state / (D + 1);
      const uint32_t f = state % (D + 1);
      uint64_t flip = f ? (1ull << (f - 1)) : 0ull;
      for (--lvl; lvl >= 0; --lvl) {
        uint32_t g = 0;
#pragma unroll
        for (int d = 0; d < D; ++d) g |= ((c[d] >> lvl) & 1u) << d;
        key = (key << D) | hilbert_step<D>(g, rot, flip);
      }
      // hilbert_finish; shifts past the key's top bit change nothing
      key ^= low_bits;
#pragma unroll
      for (int sh = 1; sh < 64; sh *= 2) key ^= key >> sh;
    } else {
      int64_t c[D];
#pragma unroll
      for (int d = 0; d < D; ++d) c[d] = quantise(p[d], bits, mode);
      key = hilbert_index_t<D>(bits, c);
    }
    keys[i] = key;
    most = max(most, key);
  }
  for (int o = 16; o > 0; o >>= 1) most = max(most, (uint64_t)__shfl_xor_sync(0xffffffffu, (unsigned long long)most, o));
  if ((threadIdx.x & 31) == 0 && most) atomicMax(max_key, (unsigned long long)most);
}

// ---------------------------------------------------------------------------
// Radix sort of (key, position), 8-bit digits, least significant first: one
// histogram pass for all digits, then one sweep per digit that reads and
// writes every pair once ("Onesweep", A. Adinets and D. Merrill, 2022; the
// tiles' prefixes by decoupled look-back, D. Merrill and M. Garland,
// "Single-pass Parallel Prefix Scan with Decoupled Look-back", 2016).
//
// Keys of more than 32 bits are first sorted by the 32 bits below their
// highest set bit only (four sweeps): n objects rarely share many of those.
// k_rs_ties and k_rs_runs then order every run of equal top bits by the
// rest, in place (a thread, a warp or a CTA per run); a run that cannot be
// sets a flag, and only then do the sweeps over all digits
// that follow do anything.  Where objects lie close to one another many share
// their top bits and the ties cost more than the four sweeps they save (16 M
// objects in 64 clusters of deviation 0.005: 0.66 ms, 0.002: all twelve
// sweeps), so large sorts sample the keys first and leave such to the sweeps
// over all digits.  Bound by issue (ranking a pair) and the
// pairs' traffic, 24 bytes per pair and sweep.  16 M pairs of 63 bits: an
// upsweep, table scan and downsweep per digit, 8 digits, 1,284 us; this
// 750-860 us (150 us a sweep), 1.3 ms over all digits, 2.2 ms where a run too
// long for its place was not seen by the sample.
// ---------------------------------------------------------------------------
constexpr int RS_THREADS = 256;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_ITEMS = 12;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_PER_WARP = RS_TILE / RS_WARPS;
constexpr uint32_t RS_MAX_PASSES = 8;
constexpr uint32_t RS_TOP = 4;          // sweeps over the top bits
constexpr uint32_t kRunSort = 2048;     // pairs of a run that a CTA sorts in shared memory
constexpr uint32_t kRunCap = 1u << 18;  // longest run of equal top bits that is ordered in place
constexpr uint32_t RS_POLLS = 1u << 22; // polls of the earlier tiles' statuses before a tile gives up
constexpr uint32_t kSortTimeout = 2;    // error bit of a tile that did

// Scratch: digit counts and tile tickets of every sweep, the
// largest key, the flag, and per tile and digit a status word: (2 sweep + 1 or
// 2) << 32 | count, odd = the tile's own count, even = the inclusive prefix.
// Statuses of earlier sweeps (and the zeros before the first) are lower than
// the current one's, so the scratch is cleared once per sort.
struct RsScratch {
  uint32_t hist[RS_TOP + RS_MAX_PASSES][256];
  uint32_t ticket[RS_TOP + RS_MAX_PASSES];
  uint32_t long_run;  // nonzero: a run of equal top bits was too long
  uint32_t nruns, nlong;  // runs listed for k_rs_runs: of up to 32 pairs, longer
  uint32_t shared;    // sampled keys that share their top bits with another one's
  uint32_t failed;    // nonzero: a tile's wait ran out
  uint32_t pad_;
  unsigned long long max_key;
};

// Whether so many objects share their top bits that the sweeps over all digits
// are the cheaper way from the start (tight: of more than this many sampled).
__device__ __forceinline__ bool rs_tight(const RsScratch* rs, uint32_t tight) { return rs->shared > tight; }

// Whether sweep p does anything: those over the top bits unless the keys are
// tight, those over all digits if they are or a run turned out too long.
__device__ __forceinline__ bool rs_runs(const RsScratch* rs, uint32_t p, uint32_t tight) {
  const bool t = rs_tight(rs, tight);
  return p < RS_TOP ? !t : t || rs->long_run;
}

// Lowest bit of sweep p's digit: p < RS_TOP: of the top 32 bits; otherwise
// digit p - RS_TOP of the whole key.
__device__ __forceinline__ uint32_t rs_shift(const RsScratch* rs, uint32_t p) {
  if (p >= RS_TOP) return 8 * (p - RS_TOP);
  const uint32_t bits = 64u - clz64(rs->max_key);
  return (bits > 32 ? bits - 32 : 0) + 8 * p;
}
// Byte of k from bit `shift` up.
__device__ __forceinline__ uint32_t rs_digit(uint64_t k, uint32_t shift) {
  const uint32_t lo = (uint32_t)k, hi = (uint32_t)(k >> 32);
  return (shift < 32 ? __funnelshift_r(lo, hi, shift) : hi >> (shift - 32)) & 255u;
}

// Samples m keys, one at a scattered place of each n / m, and counts those
// whose top bits another sampled key has too, the rest of it being different
// (equal keys cost the ties nothing), by a hash table of 2 m zeroed words.
// Thread t of the m takes one.
__device__ __forceinline__ void rs_sample(const uint64_t* keys, uint64_t n, uint32_t m, uint32_t t, RsScratch* rs,
                                          unsigned long long* slots) {
  const uint32_t mask = 2 * m - 1;
  const uint32_t shift = rs_shift(rs, 0);
  bool shares = false;
  if (shift) {
    const uint64_t step = n / m;
    const unsigned long long k = keys[t * step + (t * 0x9e3779b1u >> 8) % step];
    const unsigned long long top = k >> shift;
    uint32_t at = (uint32_t)((top * 0x9e3779b97f4a7c15ull) >> 40) & mask;
    // (a zero word is free, so the key 0 is not counted)
    for (int probe = 0; k && probe < 16; ++probe, at = (at + 1) & mask) {
      const unsigned long long old = atomicCAS(slots + at, 0ull, k);
      if (old == 0) break;
      if (old >> shift == top) {
        shares = old != k;
        break;
      }
    }
  }
  const uint32_t c = __popc(__ballot_sync(0xffffffffu, shares));
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(&rs->shared, c);
}

// Counts of the digits of sweeps [p0, p0 + np).  The first sblocks
// blocks of the first pass take the sample instead, beside it (a kernel of its
// own: 6 to 11 us), so the pass is made whatever the sample says.
__global__ void __launch_bounds__(RS_THREADS) k_rs_hist(const uint64_t* __restrict__ keys, uint64_t n, uint32_t p0,
                                                        uint32_t np, uint32_t tight, uint32_t samples,
                                                        uint32_t sblocks, RsScratch* rs, unsigned long long* slots) {
  __shared__ uint32_t h[RS_MAX_PASSES][256];
  if (p0 >= RS_TOP && !rs_runs(rs, p0, tight)) return;
  if (blockIdx.x < sblocks) {
    for (uint32_t t = blockIdx.x * RS_THREADS + threadIdx.x; t < samples; t += sblocks * RS_THREADS)
      rs_sample(keys, n, samples, t, rs, slots);
    return;
  }
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  for (uint32_t i = tid; i < np * 256; i += RS_THREADS) (&h[0][0])[i] = 0;
  __syncthreads();
  const uint32_t shift0 = rs_shift(rs, p0);
  const uint64_t stride = (uint64_t)(gridDim.x - sblocks) * RS_THREADS;
  for (uint64_t i0 = (uint64_t)(blockIdx.x - sblocks) * RS_THREADS; i0 < n; i0 += 4 * stride) {
    uint64_t k[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const uint64_t i = i0 + u * stride + tid;
      k[u] = i < n ? __ldcs(keys + i) : 0ull;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool valid = i0 + u * stride + tid < n;
      const uint32_t act = __ballot_sync(0xffffffffu, valid);
      if (!act) break;  // warp-uniform
      for (uint32_t p = 0; p < np; ++p) {
        const uint32_t d = (uint32_t)(k[u] >> (shift0 + 8 * p)) & 255u;
        // objects in spatial order share their high digits: one add per warp
        const uint32_t d0 = __shfl_sync(0xffffffffu, d, 0);
        if (act == 0xffffffffu && __all_sync(0xffffffffu, d == d0)) {
          if (lane == 0) atomicAdd(&h[p][d0], 32u);
        } else if (valid) {
          atomicAdd(&h[p][d], 1u);
        }
      }
    }
  }
  __syncthreads();
  for (uint32_t p = 0; p < np; ++p)
    if (h[p][tid]) atomicAdd(&rs->hist[p0 + p][tid], h[p][tid]);
}

__device__ __forceinline__ uint64_t ld_status(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_status(uint64_t* p, uint64_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Exclusive scan of one value per thread over a 256-thread block.
__device__ __forceinline__ uint32_t block_excl_scan256(uint32_t v, uint32_t* warp_tot) {
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t tot;
  const uint32_t ex = warp_excl_sum(v, &tot);
  if (lane == 31) warp_tot[w] = tot;
  __syncthreads();
  uint32_t before = 0;
#pragma unroll
  for (int k = 0; k < RS_WARPS; ++k) before += k < (int)w ? warp_tot[k] : 0u;
  return before + ex;
}

// One sweep.  A tile's pairs are ranked stably (the lanes of a warp with the
// same digit found by 8 ballots, one per digit bit, all lanes taking part;
// per-warp digit counters -- lane masks by shared-memory atomicOr took 33
// wavefronts per instruction), its
// digit counts published, the pairs regrouped by digit in shared memory, and
// once the look-back knows the tile's place among the earlier ones every digit
// run is written contiguously.  The slots past a short last tile's end count
// as its last pairs of digit 255 and are not written.  Tiles are taken by
// ticket, so every tile that one waits for is running or done; a wait is
// bounded all the same: after `polls` polls the tile sets kSortTimeout in *err
// and its CTA leaves without writing the tile; the sweeps that follow then do
// nothing.
__global__ void __launch_bounds__(RS_THREADS, 3) k_rs_sweep(
    const uint64_t* __restrict__ keys_in, const uint32_t* __restrict__ vals_in, uint64_t* __restrict__ keys_out,
    uint32_t* __restrict__ vals_out, uint64_t n, uint32_t ntiles, uint32_t sweep, RsScratch* rs, uint64_t* status,
    uint32_t tight, uint32_t polls, uint32_t* err) {
  __shared__ uint64_t skeys[RS_TILE];
  __shared__ uint32_t svals[RS_TILE];
  __shared__ uint32_t gofs[256];  // output position of the digit's first pair minus its slot in the tile
  __shared__ uint32_t warp_tot[RS_WARPS];
  __shared__ uint32_t s_tile;
  if (!rs_runs(rs, sweep, tight)) return;
  // the first sweep that runs: the values are the positions
  const bool first = sweep == 0 || (sweep == RS_TOP && rs_tight(rs, tight));
  // ranking counters [warp][digit], in the stage until the pairs go there
  uint32_t* wcnt = reinterpret_cast<uint32_t*>(skeys);
  static_assert(RS_WARPS * 256 <= 2 * RS_TILE, "the counters fit the stage");
  const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const uint32_t shift = rs_shift(rs, sweep);
  // first output position of this thread's digit
  const uint32_t digit0 = block_excl_scan256(rs->hist[sweep][tid], warp_tot);
  const uint32_t partial = 2 * sweep + 1, inclusive = 2 * sweep + 2;
  const uint32_t lt = lane_lt_mask();
  for (;;) {
    // (after an expired wait the pairs are incomplete: no sweep may rank them)
    if (tid == 0) s_tile = *(volatile uint32_t*)&rs->failed ? ntiles : atomicAdd(&rs->ticket[sweep], 1u);
    for (uint32_t i = tid; i < RS_WARPS * 256; i += RS_THREADS) wcnt[i] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile >= ntiles) return;
    const uint64_t base = (uint64_t)tile * RS_TILE;
    const uint32_t tile_n = (uint32_t)((n - base) < (uint64_t)RS_TILE ? (n - base) : RS_TILE);
    uint64_t k[RS_ITEMS];
    uint32_t v[RS_ITEMS];
    uint32_t pos[RS_ITEMS];
    // every load of the tile in flight before the first ranking step
    const uint32_t l0 = w * RS_PER_WARP + lane;
    if (tile_n == RS_TILE) {
#pragma unroll
      for (int r = 0; r < RS_ITEMS; ++r) k[r] = __ldcs(keys_in + base + l0 + r * 32);
#pragma unroll
      for (int r = 0; r < RS_ITEMS; ++r)
        v[r] = first ? (uint32_t)base + l0 + r * 32 : __ldcs(vals_in + base + l0 + r * 32);
    } else {
#pragma unroll
      for (int r = 0; r < RS_ITEMS; ++r) {
        const uint32_t li = l0 + r * 32;
        k[r] = li < tile_n ? __ldcs(keys_in + base + li) : ~0ull;
        v[r] = (uint32_t)base + li;
        if (!first && li < tile_n) v[r] = __ldcs(vals_in + base + li);
      }
    }
    uint32_t* wc = wcnt + w * 256;
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
      const uint32_t d = rs_digit(k[r], shift);
      uint32_t peers = 0xffffffffu;  // lanes with the same digit
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t bal = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? bal : ~bal;
      }
      const uint32_t prev = wc[d];
      pos[r] = prev + __popc(peers & lt);
      __syncwarp();
      if ((peers & lt) == 0) wc[d] = prev + __popc(peers);  // the first of them
      __syncwarp();
    }
    __syncthreads();
    // thread = digit: counts across the warps, published
    uint32_t c[RS_WARPS], count = 0;
#pragma unroll
    for (int ww = 0; ww < RS_WARPS; ++ww) {
      c[ww] = wcnt[ww * 256 + tid];
      count += c[ww];
    }
    const uint32_t real = tid == 255 ? count - (RS_TILE - tile_n) : count;
    uint64_t* mine = status + (uint64_t)tile * 256 + tid;
    st_status(mine, (uint64_t)(tile == 0 ? inclusive : partial) << 32 | real);
    const uint32_t ex = block_excl_scan256(count, warp_tot);
    // first slot of (digit, warp) in the tile
    uint32_t run = ex;
#pragma unroll
    for (int ww = 0; ww < RS_WARPS; ++ww) {
      wcnt[ww * 256 + tid] = run;
      run += c[ww];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) pos[r] += wc[rs_digit(k[r], shift)];
    __syncthreads();  // the counters are read; the pairs take their place
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
      skeys[pos[r]] = k[r];
      svals[pos[r]] = v[r];
    }
    // look-back: counts of the digit in the earlier tiles, four statuses at a time
    uint32_t before = 0;
    bool gave_up = false;
    if (tile) {
      int64_t t = (int64_t)tile - 1;
      uint32_t spins = 0;
      bool done = false;
      while (!done) {
        uint64_t st[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          st[j] = t - j >= 0 ? ld_status(status + (uint64_t)(t - j) * 256 + tid) : (uint64_t)inclusive << 32;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (done || (uint32_t)(st[j] >> 32) < partial) break;
          before += (uint32_t)st[j];
          done = (uint32_t)(st[j] >> 32) == inclusive;
          --t;
        }
        if (!done && ++spins > polls) {
          rs->failed = 1;
          atomicOr(err, kSortTimeout);
          done = gave_up = true;
        }
      }
      if (!gave_up) st_status(mine, (uint64_t)inclusive << 32 | (before + real));
    }
    gofs[tid] = digit0 + before - ex;
    if (__syncthreads_or(gave_up)) return;
#pragma unroll 4
    for (uint32_t i = tid; i < tile_n; i += RS_THREADS) {
      const uint64_t key = skeys[i];
      const uint32_t dst = gofs[rs_digit(key, shift)] + i;
      keys_out[dst] = key;
      vals_out[dst] = svals[i];
    }
    __syncthreads();  // the stage is free for the next tile
  }
}

// Orders every run of equal top bits by the whole key (equal keys keep their
// order): the thread at a run's start swaps a pair, or lists the run for
// k_rs_runs.  Other threads only compare their key with the one before.
// (Insertion by one thread up to 32 keys took 148 us on 16 M clustered points:
// a chain of dependent reads per step.)
__global__ void k_rs_ties(uint64_t* keys, uint32_t* vals, uint64_t n, RsScratch* rs, uint2* runs, uint64_t cap,
                          uint32_t tight) {
  if (rs_tight(rs, tight)) return;
  const uint32_t shift = rs_shift(rs, 0);
  if (shift == 0) return;  // the top bits were all of them
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i + 1 < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t k0 = keys[i], k1 = keys[i + 1], top = k0 >> shift;
    if ((k1 >> shift) != top) continue;
    // out of order in a run that is longer than kRunCap, or half of it (there
    // is a key half the length away): runs of equal keys only pass, whatever
    // their length
    if (k0 > k1 && ((i >= kRunCap / 2 && (keys[i - kRunCap / 2] >> shift) == top) ||
                    (i + kRunCap / 2 < n && (keys[i + kRunCap / 2] >> shift) == top)))
      rs->long_run = 1;
    if (i > 0 && (keys[i - 1] >> shift) == top) continue;
    if (i + 2 >= n || (keys[i + 2] >> shift) != top) {
      if (k0 > k1) {
        const uint32_t v0 = vals[i], v1 = vals[i + 1];
        keys[i] = k1, keys[i + 1] = k0;
        vals[i] = v1, vals[i + 1] = v0;
      }
      continue;
    }
    // the end by steps of twice the length, then by halving
    uint64_t in = i + 2, out = min(n, i + 6);  // in the run; past it or not known
    while (out < n && out - i <= kRunCap && (keys[out] >> shift) == top) {
      in = out;
      out = min(n, i + 2 * (out - i));
    }
    while (out - in > 1) {
      const uint64_t mid = in + (out - in) / 2;
      if ((keys[mid] >> shift) == top) in = mid;
      else out = mid;
    }
    const uint32_t len = (uint32_t)(out - i);
    if (len > kRunCap) continue;
    if (len <= 32) runs[atomicAdd(&rs->nruns, 1u)] = make_uint2((uint32_t)i, len);
    else runs[cap - 1 - atomicAdd(&rs->nlong, 1u)] = make_uint2((uint32_t)i, len);
  }
}

// Bitonic sort by (key, value) of the cnt <= kRunSort pairs in shared memory.
__device__ __forceinline__ void sort_in_smem(uint64_t* sk, uint32_t* sv, uint32_t cnt) {
  uint32_t len = 64;
  while (len < cnt) len *= 2;
  for (uint32_t i = cnt + threadIdx.x; i < len; i += RS_THREADS) sk[i] = ~0ull, sv[i] = 0xffffffffu;  // last
  __syncthreads();
  for (uint32_t size = 2; size <= len; size *= 2) {
    for (uint32_t step = size / 2; step > 0; step /= 2) {
      for (uint32_t t = threadIdx.x; t < len / 2; t += RS_THREADS) {
        const uint32_t a = 2 * step * (t / step) + t % step, b = a + step;
        const uint64_t ka = sk[a], kb = sk[b];
        const uint32_t va = sv[a], vb = sv[b];
        const bool up = (a & size) == 0;
        if ((ka > kb || (ka == kb && va > vb)) == up) {
          sk[a] = kb, sk[b] = ka;
          sv[a] = vb, sv[b] = va;
        }
      }
      __syncthreads();
    }
  }
}

// The listed runs; the values of a run ascend before it is ordered, so order
// by (key, value) keeps equal keys as they are.
//   up to 32 pairs (the list's front): a warp ranks every pair among the others;
//   up to kRunSort pairs: a CTA sorts them in shared memory;
//   more: a run is this long where many objects coincide (points clamped to
//   a corner of the domain), so the CTA sorts the pairs below and above the
//   middle pair's key and moves those equal to it between them, through ktmp
//   and vtmp.
//   Where they are not few the flag is set instead.
__global__ void __launch_bounds__(RS_THREADS) k_rs_runs(uint64_t* keys, uint32_t* vals, uint64_t* ktmp,
                                                        uint32_t* vtmp, RsScratch* rs,
                                                        const uint2* __restrict__ runs, uint64_t cap) {
  __shared__ uint64_t sk[kRunSort];
  __shared__ uint32_t sv[kRunSort];
  __shared__ uint32_t warp_tot[RS_WARPS];
  __shared__ uint32_t s_cnt[3];
  const uint32_t tid = threadIdx.x, lane = tid & 31;
  for (uint32_t r = (blockIdx.x * RS_THREADS + tid) >> 5; r < rs->nruns; r += gridDim.x * RS_WARPS) {
    const uint2 run = runs[r];
    const bool mine = lane < run.y;
    const uint64_t k = mine ? keys[run.x + lane] : ~0ull;
    const uint32_t v = mine ? vals[run.x + lane] : 0u;
    uint32_t rank = 0;
    for (uint32_t j = 0; j < run.y; ++j) {
      const uint64_t kj = __shfl_sync(0xffffffffu, (unsigned long long)k, j);
      rank += kj < k || (kj == k && j < lane);
    }
    if (mine) {
      keys[run.x + rank] = k;
      vals[run.x + rank] = v;
    }
  }
  for (uint32_t r = blockIdx.x; r < rs->nlong; r += gridDim.x) {
    const uint2 run = runs[cap - 1 - r];
    uint64_t* rk = keys + run.x;
    uint32_t* rv = vals + run.x;
    __syncthreads();
    if (run.y <= kRunSort) {
      for (uint32_t i = tid; i < run.y; i += RS_THREADS) sk[i] = rk[i], sv[i] = rv[i];
      sort_in_smem(sk, sv, run.y);
      for (uint32_t i = tid; i < run.y; i += RS_THREADS) rk[i] = sk[i], rv[i] = sv[i];
      continue;
    }
    const uint64_t pivot = rk[run.y / 2];
    if (tid < 3) s_cnt[tid] = 0;
    __syncthreads();
    uint32_t below = 0, above = 0;
    for (uint32_t i = tid; i < run.y; i += RS_THREADS) {
      const uint64_t k = rk[i];
      below += k < pivot;
      above += k > pivot;
    }
    if (below) atomicAdd(&s_cnt[0], below);
    if (above) atomicAdd(&s_cnt[1], above);
    __syncthreads();
    below = s_cnt[0], above = s_cnt[1];
    if (below > kRunSort || above > kRunSort) {
      if (tid == 0) rs->long_run = 1;
      continue;
    }
    if (below + above == 0) continue;
    // the equal ones' values, compacted behind the `below` places, into vtmp
    uint32_t seen = 0;  // pairs not equal to the pivot so far
    for (uint32_t i0 = 0; i0 < run.y; i0 += RS_THREADS * 8) {
      uint32_t other = 0, m = 0;
#pragma unroll
      for (uint32_t u = 0; u < 8; ++u) {
        const uint32_t i = i0 + tid * 8 + u;
        if (i < run.y && rk[i] != pivot) m |= 1u << u;
      }
      other = __popc(m);
      uint32_t nb = seen + block_excl_scan256(other, warp_tot);
#pragma unroll
      for (uint32_t u = 0; u < 8; ++u) {
        const uint32_t i = i0 + tid * 8 + u;
        if (i >= run.y) break;
        if ((m >> u) & 1u) ++nb;
        else vtmp[run.x + below + i - nb] = rv[i];
      }
#pragma unroll
      for (int w = 0; w < RS_WARPS; ++w) seen += warp_tot[w];
      __syncthreads();
    }
    // the others, one side at a time: gathered, sorted, to their places in ktmp and vtmp
    for (uint32_t side = 0; side < 2; ++side) {
      const uint32_t cnt = side ? above : below, base = side ? run.y - above : 0u;
      if (tid == 0) s_cnt[2] = 0;
      __syncthreads();
      for (uint32_t i = tid; i < run.y; i += RS_THREADS) {
        const uint64_t k = rk[i];
        if (side ? k > pivot : k < pivot) {
          const uint32_t at = atomicAdd(&s_cnt[2], 1u);
          sk[at] = k;
          sv[at] = rv[i];
        }
      }
      sort_in_smem(sk, sv, cnt);
      for (uint32_t i = tid; i < cnt; i += RS_THREADS) {
        ktmp[run.x + base + i] = sk[i];
        vtmp[run.x + base + i] = sv[i];
      }
      __syncthreads();
    }
    for (uint32_t i = tid; i < run.y; i += RS_THREADS) {
      rk[i] = i >= below && i < run.y - above ? pivot : ktmp[run.x + i];
      rv[i] = vtmp[run.x + i];
    }
  }
}

// Generic exclusive scan of uint32 (3 kernels: chunk sums, scan of sums, apply).
constexpr int SC_THREADS = 256;
constexpr int SC_ITEMS = 16;
constexpr int SC_CHUNK = SC_THREADS * SC_ITEMS;

template <class T>
__device__ __forceinline__ T warp_incl_scan(T x) {
  const uint32_t lane = threadIdx.x & 31;
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  return x;
}

template <class T>
__device__ T block_excl_scan(T v, T* warp_tot, T* total) {
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t nw = blockDim.x >> 5;
  T x = warp_incl_scan(v);
  if (lane == 31) warp_tot[w] = x;
  __syncthreads();
  if (w == 0) {
    T t = (lane < nw) ? warp_tot[lane] : (T)0;
    t = warp_incl_scan(t);
    if (lane < nw) warp_tot[lane] = t;
  }
  __syncthreads();
  T before = (w > 0) ? warp_tot[w - 1] : (T)0;
  if (total) *total = warp_tot[nw - 1];
  __syncthreads();
  return before + x - v;
}

template <class T>
__global__ void k_scan_sums(const T* __restrict__ in, uint64_t n, T* __restrict__ sums) {
  __shared__ T wt[32];
  const uint64_t base = (uint64_t)blockIdx.x * SC_CHUNK;
  T s = 0;
  for (int r = 0; r < SC_ITEMS; ++r) {
    uint64_t i = base + (uint64_t)r * SC_THREADS + threadIdx.x;
    if (i < n) s += in[i];
  }
  T total;
  block_excl_scan(s, wt, &total);
  if (threadIdx.x == 0) sums[blockIdx.x] = total;
}

template <class T>
__global__ void k_scan_partials(T* sums, uint32_t m, T* grand_total) {
  __shared__ T wt[32];
  __shared__ T carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t b = 0; b < m; b += blockDim.x) {
    uint32_t i = b + threadIdx.x;
    T v = (i < m) ? sums[i] : (T)0;
    T tot;
    T ex = block_excl_scan(v, wt, &tot);
    if (i < m) sums[i] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0 && grand_total) *grand_total = carry;
}

template <class T>
__global__ void k_scan_apply(const T* __restrict__ in, T* __restrict__ out, uint64_t n,
                             const T* __restrict__ sums) {
  __shared__ T wt[32];
  const uint64_t base = (uint64_t)blockIdx.x * SC_CHUNK + (uint64_t)threadIdx.x * SC_ITEMS;
  T vals[SC_ITEMS];
  T s = 0;
#pragma unroll
  for (int r = 0; r < SC_ITEMS; ++r) {
    uint64_t i = base + r;
    vals[r] = (i < n) ? in[i] : (T)0;
    s += vals[r];
  }
  T ex = block_excl_scan(s, wt, (T*)nullptr) + sums[blockIdx.x];
#pragma unroll
  for (int r = 0; r < SC_ITEMS; ++r) {
    uint64_t i = base + r;
    if (i < n) out[i] = ex;
    ex += vals[r];
  }
}

// The whole scan in one CTA: up to SC_ONE values, 16 consecutive ones per
// thread.  Short scans are launch-bound: three kernels of 2 us each and their
// gaps against one of 3.
constexpr uint64_t SC_ONE = 1024 * SC_ITEMS;
template <class T>
__global__ void __launch_bounds__(1024) k_scan_one(const T* __restrict__ in, T* __restrict__ out, uint32_t n,
                                                   T* grand_total) {
  __shared__ T wt[32];
  const uint32_t base = threadIdx.x * SC_ITEMS;
  T vals[SC_ITEMS];
  T s = 0;
#pragma unroll
  for (int r = 0; r < SC_ITEMS; ++r) {
    vals[r] = base + r < n ? in[base + r] : (T)0;
    s += vals[r];
  }
  T total;
  T ex = block_excl_scan(s, wt, &total);
#pragma unroll
  for (int r = 0; r < SC_ITEMS; ++r) {
    if (base + r < n) out[base + r] = ex;
    ex += vals[r];
  }
  if (threadIdx.x == 0 && grand_total) *grand_total = total;
}

// objs -> sorted SoA arrays and the leaves' MBRs; flags non-finite coordinates
// in *bad (bit 1).  The permutation of a sort that timed out holds anything,
// so positions are bounded.  *inverted: see qcp_index.  A block packs blockDim.x / fanout whole leaves at a time, one
// object per thread, so a leaf's MBR comes from registers: every warp reduces
// its 32 objects (as order-preserving integers), the leaf's warps meet in
// shared memory.  Bound by the gather of whole rows in key order; the separate
// pass over the packed coordinates that it replaces took 87 us of 2.04 ms for
// 16 M 3-D points, 620 us for 32 M 8-D rectangles.  V: floats per load of a row.
__device__ __forceinline__ uint32_t order_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float from_order_key(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

template <int NC, int V>
__device__ __forceinline__ void load_row(float (&x)[NC], const float* o) {
#pragma unroll
  for (int c = 0; c < NC; c += V) {
    if constexpr (V == 4) {
      const float4 t = __ldg(reinterpret_cast<const float4*>(o + c));
      x[c] = t.x, x[c + 1] = t.y, x[c + 2] = t.z, x[c + 3] = t.w;
    } else if constexpr (V == 2) {
      const float2 t = __ldg(reinterpret_cast<const float2*>(o + c));
      x[c] = t.x, x[c + 1] = t.y;
    } else {
      x[c] = __ldg(o + c);
    }
  }
}

template <int D, bool RECT, int V>
__global__ void __launch_bounds__(256) k_pack(const float* __restrict__ objs, const uint32_t* __restrict__ perm,
                                              uint64_t n, uint64_t npad, uint32_t fanout, uint64_t nleaves,
                                              uint64_t pad0, float* __restrict__ coords, int32_t* __restrict__ ids,
                                              float* __restrict__ mbr, uint32_t* bad, uint32_t* inverted) {
  constexpr int NC = RECT ? 2 * D : D;
  __shared__ uint32_t wlo[8][D], whi[8][D];
  const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const uint32_t per = blockDim.x / fanout;  // leaves per block and round
  for (uint64_t j0 = (uint64_t)blockIdx.x * per; j0 < pad0; j0 += (uint64_t)gridDim.x * per) {
    const uint64_t i = j0 * fanout + tid;
    uint32_t lo[D], hi[D];
#pragma unroll
    for (int d = 0; d < D; ++d) lo[d] = 0xffffffffu, hi[d] = 0u;
    if (i < npad) {
      float x[NC];
      if (i < n) {
        const uint32_t id = min(__ldcs(perm + i), (uint32_t)n - 1);
        load_row<NC, V>(x, objs + (uint64_t)id * NC);
        bool finite = true;
#pragma unroll
        for (int c = 0; c < NC; ++c) finite &= isfinite(x[c]);
        if (!finite) atomicOr(bad, 1u);
        if constexpr (RECT) {
          bool inv = false;
#pragma unroll
          for (int d = 0; d < D; ++d) inv |= x[d] > x[D + d];
          if (inv) *inverted = 1;
        }
        ids[i] = (int32_t)id;
#pragma unroll
        for (int d = 0; d < D; ++d) {
          lo[d] = order_key(x[d]);
          hi[d] = order_key(x[RECT ? D + d : d]);
        }
      } else {
#pragma unroll
        for (int c = 0; c < NC; ++c) x[c] = __int_as_float(0x7fc00000);
        ids[i] = -1;
      }
#pragma unroll
      for (int c = 0; c < NC; ++c) coords[(uint64_t)c * npad + i] = x[c];
    }
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const uint32_t a = __reduce_min_sync(0xffffffffu, lo[d]), b = __reduce_max_sync(0xffffffffu, hi[d]);
      if (lane == 0) wlo[w][d] = a, whi[w][d] = b;
    }
    __syncthreads();
    // one thread per (leaf, MBR component); past the last leaf: empty
    for (uint32_t e = tid; e < per * 2 * D; e += blockDim.x) {
      const uint32_t lf = e / (2 * D), c = e % (2 * D);
      const uint64_t j = j0 + lf;
      if (j >= pad0) continue;
      const uint32_t w0 = lf * (fanout >> 5), w1 = w0 + (fanout >> 5);
      float m = c < D ? INFINITY : -INFINITY;
      if (j < nleaves) {
        uint32_t k = c < D ? 0xffffffffu : 0u;
        for (uint32_t ww = w0; ww < w1; ++ww) k = c < D ? min(k, wlo[ww][c]) : max(k, whi[ww][c - D]);
        m = from_order_key(k);
      }
      mbr[(uint64_t)c * pad0 + j] = m;
    }
    __syncthreads();
  }
}

__global__ void k_find_inverted(const float* __restrict__ coords, uint64_t n, uint64_t npad, uint32_t dims,
                                uint32_t* inverted) {
  for (uint32_t d = 0; d < dims; ++d) {
    const float *lo = coords + d * npad, *hi = coords + (dims + d) * npad;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
      if (lo[i] > hi[i]) *inverted = 1;
  }
}

__device__ __forceinline__ float warp_min(float x) {
  for (int o = 16; o > 0; o >>= 1) x = fminf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
__device__ __forceinline__ float warp_max(float x) {
  for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// One warp per node of level l: MBR over the children's MBRs (level l-1).
__global__ void k_level_mbr(const float* __restrict__ child, uint64_t nchild, uint64_t child_pad,
                            uint32_t dims, uint32_t fanout, uint64_t nnodes, uint64_t pad,
                            float* __restrict__ mbr) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t k = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; k < pad; k += warps) {
    if (k >= nnodes) {
      if (lane < dims) {
        mbr[(uint64_t)lane * pad + k] = INFINITY;
        mbr[(uint64_t)(dims + lane) * pad + k] = -INFINITY;
      }
      continue;
    }
    const uint64_t c0 = k * fanout;
    const uint64_t c1 = (c0 + fanout < nchild) ? c0 + fanout : nchild;
    for (uint32_t d = 0; d < dims; ++d) {
      float lo = INFINITY, hi = -INFINITY;
      for (uint64_t c = c0 + lane; c < c1; c += 32) {
        lo = fminf(lo, child[(uint64_t)d * child_pad + c]);
        hi = fmaxf(hi, child[(uint64_t)(dims + d) * child_pad + c]);
      }
      lo = warp_min(lo);
      hi = warp_max(hi);
      if (lane == 0) {
        mbr[(uint64_t)d * pad + k] = lo;
        mbr[(uint64_t)(dims + d) * pad + k] = hi;
      }
    }
  }
}

uint32_t grid_for(uint64_t work, uint32_t per_block, uint32_t cap_blocks) {
  uint64_t g = (work + per_block - 1) / per_block;
  if (g < 1) g = 1;
  if (g > cap_blocks) g = cap_blocks;
  return (uint32_t)g;
}

}  // namespace

int num_sms() {
  static int sms = 0;
  if (!sms) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
      sms = 148;
  }
  return sms;
}

size_t scan_scratch_bytes(uint64_t n) {
  return sizeof(uint64_t) * (size_t)((n + SC_CHUNK - 1) / SC_CHUNK + 1);
}

// The chunk sums live in `scratch` when the caller passes one (at least
// scan_scratch_bytes(n) bytes), else in a stream-ordered temporary.  Captured
// pipelines pass scratch: a temporary would become a graph memory node,
// whose physical memory the driver maps at a launch that needs more of it
// than the graphs already running hold.
template <class T>
qcp_status exclusive_scan(const T* in, T* out, uint64_t n, T* grand_total, DevPool& pool,
                          cudaStream_t s, void* scratch, size_t scratch_bytes) {
  (void)pool;
  if (n && n <= SC_ONE) {
    // no more threads than hold a value, in whole warps
    const uint32_t threads = (uint32_t)(((n + SC_ITEMS - 1) / SC_ITEMS + 31) & ~31ull);
    k_scan_one<T><<<1, threads, 0, s>>>(in, out, (uint32_t)n, grand_total);
    note_launch();
    return check_launch("exclusive_scan");
  }
  const uint32_t nblk = (uint32_t)((n + SC_CHUNK - 1) / SC_CHUNK);
  void* sums = scratch;
  if (scratch) {
    if (scratch_bytes < sizeof(T) * (nblk ? nblk : 1)) {
      set_error("exclusive_scan: scratch too small");
      return QCP_ERR_BAD_ARG;
    }
  } else {
    QCP_TRY(temp_alloc(sizeof(T) * (nblk ? nblk : 1), s, &sums));
  }
  if (n) {
    k_scan_sums<T><<<nblk, SC_THREADS, 0, s>>>(in, n, (T*)sums);
    k_scan_partials<T><<<1, 1024, 0, s>>>((T*)sums, nblk, grand_total);
    k_scan_apply<T><<<nblk, SC_THREADS, 0, s>>>(in, out, n, (T*)sums);
    note_launch(3);
  }
  qcp_status st = check_launch("exclusive_scan");
  if (!scratch) temp_free(sums, s);
  return st;
}

template qcp_status exclusive_scan<uint32_t>(const uint32_t*, uint32_t*, uint64_t, uint32_t*,
                                             DevPool&, cudaStream_t, void*, size_t);
template qcp_status exclusive_scan<uint64_t>(const uint64_t*, uint64_t*, uint64_t, uint64_t*,
                                             DevPool&, cudaStream_t, void*, size_t);

template <int D>
static qcp_status launch_keys(const float* objs, uint64_t n, uint32_t is_rect, uint32_t key_mode, uint32_t key_bits,
                              uint64_t* keys, unsigned long long* max_key, cudaStream_t s) {
  const size_t smem = key_mode == QCP_KEY_NORM && D > 1 ? sizeof(uint16_t) * hilbert_tab_size<D>() : 0;
  // (a block fills its table first: no more blocks than are resident)
  k_keys<D><<<grid_for(n, 256, num_sms() * (smem > 16384 ? 4 : 8)), 256, smem, s>>>(objs, n, is_rect, key_mode,
                                                                                   key_bits, keys, max_key);
  note_launch();
  return check_launch("k_keys");
}

qcp_status build_keys(const float* objs, uint64_t n, uint32_t dims, uint32_t is_rect,
                      uint32_t key_mode, uint32_t key_bits, uint64_t* keys, uint64_t* max_key, cudaStream_t s) {
  QCP_CUDA(cudaMemsetAsync(max_key, 0, sizeof(uint64_t), s));
  qcp_status st = QCP_OK;
  QCP_DISPATCH_D(dims, st = launch_keys<DD>(objs, n, is_rect, key_mode, key_bits, keys, (unsigned long long*)max_key, s));
  return st;
}

namespace {
thread_local uint32_t t_sort_polls = RS_POLLS;
}
// For tests: most polls of a wait in the sorts that this host thread launches
// (negative: the default).  Not part of the ABI.
extern "C" void qcp_test_sort_polls(int polls) { t_sort_polls = polls < 0 ? RS_POLLS : (uint32_t)polls; }

static uint64_t rs_run_cap(uint64_t n) { return n / 3 + 1; }  // runs of three pairs at least

// Objects from which the sort of long keys samples them first, and how many it
// takes (of 1 M objects 65,536 cost a rebuild of 202 us 14, 16,384 two).
constexpr uint64_t kSampleMin = 1u << 19;
static uint32_t rs_samples(uint64_t n) { return n < kSampleMin ? 0u : (n < (1u << 23) ? 1u << 14 : 1u << 16); }

// The sample's limit: what it counts where every object shares its top bits
// with x n / m others (m samples in cells of x each).  From 2^21 objects 1.6
// others: rebuilds of 16 M objects with 1, 2 and 4 of them take 1.94, 2.20 and
// 2.29 ms by top bits and ties, 2.01 by all digits, of 4 M 0.55, 0.60 and 0.63
// against 0.60.  Fewer objects leave the sweeps launch-bound, and only long
// runs cost more than they do: 1 M objects with 4 and 1,000 others 0.25 and
// 0.34 ms against 0.27.
static uint32_t rs_tight_limit(uint64_t n) {
  const double m = rs_samples(n), x = (n < (1u << 21) ? 16 : 1.6) * m / (double)n;
  return m ? (uint32_t)(m * (1 + std::expm1(-x) / x)) : 0xffffffffu;
}

size_t radix_scratch_bytes(uint64_t n) {
  return sizeof(RsScratch) + sizeof(uint64_t) * 256 * (size_t)((n + RS_TILE - 1) / RS_TILE) +
         sizeof(uint64_t) * 2 * rs_samples(n) + sizeof(uint2) * (size_t)rs_run_cap(n);
}

qcp_status radix_sort_pairs(uint64_t* keys, uint32_t* vals, uint64_t* keys_tmp, uint32_t* vals_tmp,
                            uint64_t n, uint32_t key_bits, const uint64_t* max_key, uint32_t* err, cudaStream_t s,
                            bool* result_in_tmp, void* scratch, size_t scratch_bytes) {
  *result_in_tmp = false;
  if (n <= 1) {
    QCP_CUDA(cudaMemsetAsync(vals, 0, sizeof(uint32_t), s));
    return QCP_OK;
  }
  const uint32_t ntiles = (uint32_t)((n + RS_TILE - 1) / RS_TILE);
  const size_t need = radix_scratch_bytes(n);
  void* own = nullptr;
  if (scratch) {
    // caller-owned scratch (a captured build): no allocation on the stream
    if (scratch_bytes < need) {
      set_error("radix_sort_pairs: scratch too small");
      return QCP_ERR_BAD_ARG;
    }
  } else {
    QCP_TRY(temp_alloc(need, s, &own));
    scratch = own;
  }
  RsScratch* rs = static_cast<RsScratch*>(scratch);
  uint64_t* status = reinterpret_cast<uint64_t*>(rs + 1);
  uint64_t* slots = status + (size_t)ntiles * 256;
  uint2* runs = reinterpret_cast<uint2*>(slots + 2 * rs_samples(n));
  const uint32_t tight = rs_tight_limit(n);
  const size_t clear = reinterpret_cast<char*>(runs) - static_cast<char*>(scratch);
  const uint32_t sms = num_sms();
  int fit = 1;
  qcp_status st = QCP_OK;
  if (cudaMemsetAsync(scratch, 0, clear, s) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k_rs_sweep, RS_THREADS, 0) != cudaSuccess)
    st = cuda_status(cudaGetLastError(), "radix scratch");
  const uint32_t grid = ntiles < sms * fit ? ntiles : sms * fit;
  uint64_t* kin = keys;
  uint32_t* vin = vals;  // (the first sweep's are the positions)
  uint64_t* kout = keys_tmp;
  uint32_t* vout = vals_tmp;
  // sweeps [p0, p0 + np)
  auto sweeps = [&](uint32_t p0, uint32_t np) {
    // a key per thread where the histogram is short (four in turn took twice its
    // 12 us on 1 M keys), four where the blocks are missed more (16 M)
    const uint32_t m = p0 == 0 && key_bits > 32 ? rs_samples(n) : 0, sb = m > 16384 ? m / 1024 : m / RS_THREADS;
    k_rs_hist<<<sb + grid_for(n, RS_THREADS * 8, sms * 8 - sb), RS_THREADS, 0, s>>>(
        kin, n, p0, np, tight, m, sb, rs, reinterpret_cast<unsigned long long*>(slots));
    note_launch();
    for (uint32_t p = p0; p < p0 + np; ++p) {
      k_rs_sweep<<<grid, RS_THREADS, 0, s>>>(kin, vin, kout, vout, n, ntiles, p, rs, status, tight, t_sort_polls,
                                             err);
      note_launch();
      kin = kout;
      vin = vout;
      *result_in_tmp = !*result_in_tmp;
      kout = *result_in_tmp ? keys : keys_tmp;
      vout = *result_in_tmp ? vals : vals_tmp;
    }
  };
  if (st == QCP_OK) {
    if (key_bits > 32) {
      cudaMemcpyAsync(&rs->max_key, max_key, sizeof(uint64_t), cudaMemcpyDeviceToDevice, s);
      sweeps(0, RS_TOP);
      k_rs_ties<<<grid_for(n, 256, sms * 16), 256, 0, s>>>(keys, vals, n, rs, runs, rs_run_cap(n), tight);
      k_rs_runs<<<sms * 4, RS_THREADS, 0, s>>>(keys, vals, keys_tmp, vals_tmp, rs, runs, rs_run_cap(n));
      note_launch(2);
      // all digits, if a run was too long; an even number of sweeps, so that
      // the result is where it is without them
      sweeps(RS_TOP, ((key_bits + 15) / 16) * 2);
    } else {
      sweeps(0, (key_bits + 7) / 8);
    }
    st = check_launch("radix_sort_pairs");
  }
  if (own) temp_free(own, s);
  return st;
}

template <int D, bool RECT>
static void launch_pack(qcp_index* ix, const float* objs, const uint32_t* perm, cudaStream_t s, uint32_t* d_bad) {
  const uint32_t F = ix->fanout, per = 256 / F;
  const uint32_t grid = grid_for(ix->level_pad[0], per, num_sms() * 16);
  // rows are loaded in pieces that divide them and that objs is aligned to
  constexpr int NC = RECT ? 2 * D : D;
  constexpr int V = NC % 4 == 0 ? 4 : (NC % 2 == 0 ? 2 : 1);
  const bool wide = reinterpret_cast<uintptr_t>(objs) % (sizeof(float) * V) == 0;
  auto* kern = wide ? k_pack<D, RECT, V> : k_pack<D, RECT, 1>;
  kern<<<grid, per * F, 0, s>>>(objs, perm, ix->n, ix->npad, F, ix->level_nodes[0], ix->level_pad[0], ix->coords,
                                ix->ids, ix->mbr[0], d_bad, ix->inverted);
}

qcp_status build_pack(qcp_index* ix, const float* objs, const uint32_t* perm, cudaStream_t s,
                      uint32_t* d_bad) {
  if (ix->is_rect) QCP_CUDA(cudaMemsetAsync(ix->inverted, 0, sizeof(uint32_t), s));
  QCP_DISPATCH_D(ix->dims, if (ix->is_rect) launch_pack<DD, true>(ix, objs, perm, s, d_bad);
                 else launch_pack<DD, false>(ix, objs, perm, s, d_bad));
  note_launch();
  return check_launch("k_pack");
}

qcp_status find_inverted(qcp_index* ix, cudaStream_t s) {
  if (!ix->is_rect) return QCP_OK;
  QCP_CUDA(cudaMemsetAsync(ix->inverted, 0, sizeof(uint32_t), s));
  k_find_inverted<<<grid_for(ix->n, 256, num_sms() * 8), 256, 0, s>>>(ix->coords, ix->n, ix->npad, ix->dims,
                                                                      ix->inverted);
  note_launch();
  QCP_TRY(check_launch("k_find_inverted"));
  QCP_CUDA(cudaStreamSynchronize(s));
  return QCP_OK;
}

qcp_status build_levels(qcp_index* ix, cudaStream_t s) {
  const uint32_t threads = 256, wpb = threads / 32;
  for (uint32_t l = 1; l < ix->levels; ++l) {
    k_level_mbr<<<grid_for(ix->level_pad[l], wpb, num_sms() * 32), threads, 0, s>>>(
        ix->mbr[l - 1], ix->level_nodes[l - 1], ix->level_pad[l - 1], ix->dims, ix->fanout,
        ix->level_nodes[l], ix->level_pad[l], ix->mbr[l]);
    note_launch();
    QCP_TRY(check_launch("k_level_mbr"));
  }
  return QCP_OK;
}

qcp_status exclusive_scan_counts(const uint64_t* counts, uint64_t* offsets, uint32_t q,
                                 DevPool& pool, cudaStream_t s, void* scratch, size_t scratch_bytes) {
  // offsets has q+1 entries; offsets[q] receives the total.
  if (q == 0) {
    QCP_CUDA(cudaMemsetAsync(offsets, 0, sizeof(uint64_t), s));
    return QCP_OK;
  }
  return exclusive_scan<uint64_t>(counts, offsets, q, offsets + q, pool, s, scratch, scratch_bytes);
}

}  // namespace qcp
