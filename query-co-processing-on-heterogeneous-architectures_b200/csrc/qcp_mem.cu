// Device memory of the library: where it comes from, what stays with the
// library when it is freed, and what happens when there is none.  Host code
// only.
#include <mutex>
#include <unordered_map>
#include <vector>

#include "qcp_internal.cuh"

namespace qcp {

namespace {

constexpr int kMaxDevices = 64;

thread_local cudaStream_t t_alloc_stream = nullptr;
thread_local bool t_lasting = false;

struct Pool {
  cudaMemPool_t pool = nullptr;
  uint64_t live = 0;       // bytes allocated from it and not freed
  uint64_t threshold = 0;  // its release threshold
};
enum Kind { kPooled, kDirect, kShared };
struct Block {
  size_t bytes;
  int device;
  Kind kind;
};
struct Memory {
  std::mutex mu;
  Pool pools[kMaxDevices];
  std::unordered_map<void*, Block> blocks;       // every live allocation
  std::vector<std::pair<void*, Block>> idle;     // shared blocks that are kept, oldest first
  uint64_t idle_bytes[kMaxDevices] = {};
};
Memory& memory() {
  static Memory* m = new Memory();  // lives until exit
  return *m;
}

// The device's pool, created on first use (m.mu is held).
cudaError_t device_pool(Memory& m, int dev, Pool** out) {
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  Pool& p = m.pools[dev];
  if (!p.pool) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t made = nullptr;
    const cudaError_t e = cudaMemPoolCreate(&made, &props);
    if (e != cudaSuccess) return e;
    p.pool = made;
  }
  *out = &p;
  return cudaSuccess;
}

// The release threshold counts what is in use too, so it follows `live`: what
// the pool keeps beyond it is between 7/8 of kPoolKeeps and kPoolKeeps (the
// band saves setting it with every small buffer).  m.mu is held.
void follow(Pool& p) {
  const uint64_t most = p.live + kPoolKeeps, least = most - kPoolKeeps / 8;
  if (p.threshold >= least && p.threshold <= most) return;
  uint64_t t = most - kPoolKeeps / 16;
  if (cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &t) == cudaSuccess) p.threshold = t;
  else cudaGetLastError();
}

uint64_t reserved(const Pool& p) {
  uint64_t bytes = 0;
  if (cudaMemPoolGetAttribute(p.pool, cudaMemPoolAttrReservedMemCurrent, &bytes) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return bytes;
}

// Takes the kept shared blocks of a device off the list, the oldest first,
// until it keeps at most `keep` bytes (m.mu is held; the caller frees them).
std::vector<void*> drop_idle(Memory& m, int device, uint64_t keep) {
  std::vector<void*> out;
  for (size_t i = 0; i < m.idle.size() && m.idle_bytes[device] > keep;) {
    if (m.idle[i].second.device != device) {
      ++i;
      continue;
    }
    out.push_back(m.idle[i].first);
    m.idle_bytes[device] -= m.idle[i].second.bytes;
    m.idle.erase(m.idle.begin() + i);
  }
  return out;
}

// A kept shared block of the device for `bytes`, the smallest of at most twice
// as many.
bool take_idle(Memory& m, int device, size_t bytes, void** p) {
  std::lock_guard<std::mutex> g(m.mu);
  size_t best = m.idle.size();
  for (size_t i = 0; i < m.idle.size(); ++i) {
    const Block& b = m.idle[i].second;
    if (b.device == device && b.bytes >= bytes && b.bytes <= 2 * bytes + (1u << 20) &&
        (best == m.idle.size() || b.bytes < m.idle[best].second.bytes))
      best = i;
  }
  if (best == m.idle.size()) return false;
  *p = m.idle[best].first;
  m.blocks[*p] = m.idle[best].second;
  m.idle_bytes[device] -= m.idle[best].second.bytes;
  m.idle.erase(m.idle.begin() + best);
  return true;
}

cudaError_t allocate(void** p, size_t bytes, Kind kind, cudaStream_t s) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (!bytes) bytes = 1;
  Memory& m = memory();
  if (kind != kPooled) {
    if (kind == kShared && take_idle(m, dev, bytes, p)) return cudaSuccess;
    if ((e = cudaMalloc(p, bytes)) != cudaSuccess) return e;
    std::lock_guard<std::mutex> g(m.mu);
    m.blocks[*p] = Block{bytes, dev, kind};
    return cudaSuccess;
  }
  Pool* pool = nullptr;
  {
    std::lock_guard<std::mutex> g(m.mu);
    if ((e = device_pool(m, dev, &pool)) != cudaSuccess) return e;
  }
  if ((e = cudaMallocFromPoolAsync(p, bytes, pool->pool, s)) != cudaSuccess) return e;
  std::lock_guard<std::mutex> g(m.mu);
  m.blocks[*p] = Block{bytes, dev, kPooled};
  pool->live += bytes;
  follow(*pool);
  // If the pool holds more than the threshold although something had to be
  // added, what it keeps does not fit what is asked for now: all of it is given
  // back, or every synchronisation would release what the next call needs.
  if (reserved(*pool) > pool->threshold) cudaMemPoolTrimTo(pool->pool, pool->live);
  return cudaSuccess;
}

// As allocate; once more, without what is kept, where there is no room.
cudaError_t allocate_or_trim(void** p, size_t bytes, Kind kind, cudaStream_t s) {
  cudaError_t e = allocate(p, bytes, kind, s);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  cudaStreamSynchronize(s);  // what was freed on it is free then
  int dev = 0;
  Memory& m = memory();
  if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < kMaxDevices) {
    std::vector<void*> old;
    {
      std::lock_guard<std::mutex> g(m.mu);
      if (m.pools[dev].pool) cudaMemPoolTrimTo(m.pools[dev].pool, 0);
      old = drop_idle(m, dev, 0);
    }
    for (void* q : old) cudaFree(q);
  }
  return allocate(p, bytes, kind, s);
}

}  // namespace

cudaError_t dev_malloc_bytes(void** p, size_t bytes) {
  const bool pooled = bytes <= (t_lasting ? kPoolLargestLasting : kPoolLargest);
  return allocate_or_trim(p, bytes, pooled ? kPooled : kDirect, t_alloc_stream);
}
cudaError_t dev_malloc_shared(void** p, size_t bytes) { return allocate_or_trim(p, bytes, kShared, t_alloc_stream); }

void dev_free(void* p) {
  if (!p) return;
  Memory& m = memory();
  Block b;
  {
    std::lock_guard<std::mutex> g(m.mu);
    const auto it = m.blocks.find(p);
    if (it == m.blocks.end()) return;
    b = it->second;
    m.blocks.erase(it);
  }
  // (the calling thread's stream is one of the current device's)
  const OnDevice on(b.device);
  if (b.kind == kShared && b.bytes <= kSharedKeeps) {
    std::vector<void*> old;
    {
      std::lock_guard<std::mutex> g(m.mu);
      old = drop_idle(m, b.device, kSharedKeeps - b.bytes);
      m.idle.emplace_back(p, b);
      m.idle_bytes[b.device] += b.bytes;
    }
    for (void* q : old) cudaFree(q);
    return;
  }
  if (b.kind != kPooled) {
    cudaFree(p);
    return;
  }
  if (cudaFreeAsync(p, on.switched() ? nullptr : t_alloc_stream) != cudaSuccess) {
    cudaGetLastError();
    cudaFree(p);
  }
  std::lock_guard<std::mutex> g(m.mu);
  m.pools[b.device].live -= b.bytes;
  follow(m.pools[b.device]);
}

void dev_give_back(int device) {
  Memory& m = memory();
  if (device < 0 || device >= kMaxDevices) return;
  std::lock_guard<std::mutex> g(m.mu);
  Pool& p = m.pools[device];
  if (!p.pool) return;
  const OnDevice on(device);
  if (reserved(p) <= p.live + kPoolKeeps) return;
  cudaStreamSynchronize(on.switched() ? nullptr : t_alloc_stream);
  cudaMemPoolTrimTo(p.pool, p.live + kPoolKeeps);
}

AllocOn::AllocOn(cudaStream_t s) : before_(t_alloc_stream) { t_alloc_stream = s; }
AllocOn::~AllocOn() { t_alloc_stream = before_; }
AllocLasting::AllocLasting() { t_lasting = true; }
AllocLasting::~AllocLasting() { t_lasting = false; }

// Temporaries freed before the work that uses them has run: a buffer freed on
// one stream is handed to another stream only after the freeing stream has
// reached the free, so calls that run concurrently on different streams never
// share one.
qcp_status temp_alloc(size_t bytes, cudaStream_t s, void** out) {
  QCP_CUDA(allocate_or_trim(out, bytes, kPooled, s));
  return QCP_OK;
}

void temp_free(void* p, cudaStream_t s) {
  const AllocOn on(s);
  dev_free(p);
}

}  // namespace qcp
