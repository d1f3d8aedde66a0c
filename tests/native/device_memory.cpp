// The library's device memory (csrc/qcp_mem.cu) over a stand-in for the CUDA
// runtime's allocator that runs on the CPU.  The first argument names what is
// checked; exit code 0: it holds.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <vector>

#include "qcp_internal.cuh"

#define CHECK(c)                                          \
  do {                                                    \
    if (!(c)) {                                           \
      fprintf(stderr, "line %d: %s\n", __LINE__, #c);     \
      exit(1);                                            \
    }                                                     \
  } while (0)

constexpr uint64_t MB = 1ull << 20, GB = 1ull << 30;

// ---- the stand-in: two devices of 16 GB, a pool on each --------------------
struct FakePool {
  int device;
  uint64_t reserved = 0, used = 0, threshold = 0;
  std::vector<std::pair<void*, uint64_t>> pending;  // freed in stream order, not yet run
};
struct FakeBlock {
  uint64_t bytes;
  int device;
  FakePool* pool;
};
static int g_device = 0;
static uint64_t g_taken[2] = {0, 0};  // by cudaMalloc and by the pools
static std::map<void*, FakeBlock> g_blocks;
static std::vector<FakePool*> g_pools;
static bool g_refuse_async_free = false;
static int g_wrong_device = 0;
static uintptr_t g_next = 4096;
constexpr uint64_t kRoom = 16 * GB;

static void settle() {  // a synchronisation: pending frees are done, the pools shrink to their thresholds
  for (FakePool* p : g_pools) {
    for (auto& f : p->pending) p->used -= f.second;
    p->pending.clear();
    const uint64_t keep = p->used > p->threshold ? p->used : p->threshold;
    if (p->reserved > keep) {
      g_taken[p->device] -= p->reserved - keep;
      p->reserved = keep;
    }
  }
}

extern "C" {
cudaError_t cudaGetDevice(int* d) { return *d = g_device, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return g_device = d, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return settle(), cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
  if (g_taken[g_device] + n > kRoom) return cudaErrorMemoryAllocation;
  g_taken[g_device] += n;
  *p = reinterpret_cast<void*>(g_next += 4096);
  g_blocks[*p] = FakeBlock{n, g_device, nullptr};
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  CHECK(g_blocks.count(p));
  const FakeBlock b = g_blocks[p];
  if (b.pool) b.pool->used -= b.bytes;
  else g_taken[b.device] -= b.bytes;
  g_blocks.erase(p);
  return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps* props) {
  FakePool* f = new FakePool{props->location.id};
  g_pools.push_back(f);
  *p = reinterpret_cast<cudaMemPool_t>(f);
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void* v) {
  CHECK(a == cudaMemPoolAttrReleaseThreshold);
  reinterpret_cast<FakePool*>(p)->threshold = *static_cast<uint64_t*>(v);
  return cudaSuccess;
}
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void* v) {
  const FakePool* f = reinterpret_cast<FakePool*>(p);
  *static_cast<uint64_t*>(v) = a == cudaMemPoolAttrReservedMemCurrent ? f->reserved : f->used;
  return cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t keep) {
  FakePool* f = reinterpret_cast<FakePool*>(p);
  const uint64_t least = f->used > keep ? f->used : keep;
  if (f->reserved > least) {
    g_taken[f->device] -= f->reserved - least;
    f->reserved = least;
  }
  return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t) {
  FakePool* f = reinterpret_cast<FakePool*>(pool);
  CHECK(f->device == g_device);
  if (f->used + n > f->reserved) {
    const uint64_t more = f->used + n - f->reserved;
    if (g_taken[f->device] + more > kRoom) return cudaErrorMemoryAllocation;
    g_taken[f->device] += more;
    f->reserved += more;
  }
  f->used += n;
  *p = reinterpret_cast<void*>(g_next += 4096);
  g_blocks[*p] = FakeBlock{n, f->device, f};
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
  CHECK(g_blocks.count(p));
  const FakeBlock b = g_blocks[p];
  // (a stream of the current device)
  if (b.device != g_device || (s && b.device != 0)) ++g_wrong_device;
  if (g_refuse_async_free) return cudaErrorInvalidValue;
  CHECK(b.pool);
  b.pool->pending.emplace_back(p, b.bytes);
  g_blocks.erase(p);
  return cudaSuccess;
}
}  // extern "C"

namespace qcp {
void set_error(const std::string&) {}
qcp_status cuda_status(cudaError_t, const char*) { return QCP_ERR_CUDA; }
}  // namespace qcp

// ---- what is checked --------------------------------------------------------
using namespace qcp;

static void* get(size_t bytes) {
  void* p = nullptr;
  CHECK(dev_malloc(&p, bytes) == cudaSuccess && p);
  return p;
}

// What the pool holds and nobody uses stays within its bound after frees
// alone: no allocation follows them.
static void idle_after_frees() {
  std::vector<void*> v;
  for (int i = 0; i < 40; ++i) v.push_back(get(200 * MB));
  CHECK(g_taken[0] >= 40 * 200 * MB);
  for (void* p : v) dev_free(p);
  cudaStreamSynchronize(nullptr);
  CHECK(g_taken[0] <= kPoolKeeps);
  CHECK(g_taken[0] >= kPoolKeeps / 2);  // and it does keep some
}

// Giving back does so at once, and leaves what is in use.
static void give_back() {
  void* held = get(150 * MB);
  std::vector<void*> v;
  for (int i = 0; i < 40; ++i) v.push_back(get(200 * MB));
  for (void* p : v) dev_free(p);
  dev_give_back(0);
  CHECK(g_taken[0] <= kPoolKeeps + 150 * MB);
  dev_free(held);
}

// A buffer too large for the pool gets the room that the pool keeps.
static void large_gets_the_rest() {
  std::vector<void*> v;
  for (int i = 0; i < 8; ++i) v.push_back(get(200 * MB));
  for (void* p : v) dev_free(p);
  CHECK(g_taken[0] >= 8 * 200 * MB);
  void* large = get(kRoom - 100 * MB);
  CHECK(g_taken[0] >= kRoom - 100 * MB);
  void* p = nullptr;
  CHECK(dev_malloc(&p, 1 * GB) == cudaErrorMemoryAllocation);  // and none left is none left
  CHECK(dev_malloc(&p, 200 * MB) == cudaErrorMemoryAllocation);
  dev_free(large);
  dev_free(get(1 * GB));
}

// So does a plan's buffer, and a pool allocation of another size.
static void lasting_and_small() {
  {
    AllocLasting lasting;
    std::vector<void*> v;
    for (int i = 0; i < 400; ++i) v.push_back(get(4 * MB));
    for (void* p : v) dev_free(p);
    dev_free(get(kRoom - 10 * MB));
  }
  for (int i = 0; i < 79; ++i) get(200 * MB);
  CHECK(g_taken[0] <= kRoom);
}

// A buffer is freed on its device, in an order of its device's, whichever is
// current, and the current one stays so.
static void other_device() {
  g_device = 1;
  void* pooled = get(10 * MB);
  void* large = get(1 * GB);
  g_device = 0;
  {
    const AllocOn on(reinterpret_cast<cudaStream_t>(0x1000));  // a stream of device 0
    dev_free(pooled);
    dev_free(large);
    dev_free(get(10 * MB));
  }
  CHECK(g_device == 0);
  CHECK(g_wrong_device == 0);
  CHECK(g_blocks.empty());
}

// A refused stream-ordered free is not a leak.
static void refused_free() {
  void* p = get(10 * MB);
  g_refuse_async_free = true;
  dev_free(p);
  CHECK(g_blocks.empty());
}

// Buffers that callers see come from cudaMalloc, are kept up to a bound when
// they are freed, and serve the next such buffer of their device.
static void shared_buffers() {
  auto share = [](size_t bytes) {
    void* p = nullptr;
    CHECK(dev_malloc_shared(&p, bytes) == cudaSuccess);
    CHECK(!g_blocks[p].pool);
    return p;
  };
  void* a = share(10 * MB);
  dev_free(a);
  CHECK(share(9 * MB) == a);
  CHECK(share(9 * MB) != a);  // (in use)
  dev_free(a);
  CHECK(share(1 * MB) != a);  // not for much less
  g_device = 1;
  CHECK(share(9 * MB) != a);  // nor on another device
  g_device = 0;
  std::vector<void*> v;
  for (int i = 0; i < 60; ++i) v.push_back(share(10 * MB));
  for (void* p : v) dev_free(p);
  dev_free(share(1 * GB));
  CHECK(g_taken[0] <= kSharedKeeps + 10 * MB);
  // no room: what is kept goes first
  dev_free(share(kRoom - 15 * MB));
  CHECK(g_taken[0] <= 10 * MB);
  v.assign(1, share(200 * MB));
  dev_free(v[0]);
  {
    AllocLasting lasting;
    get(kRoom - 15 * MB);
  }
}

int main(int, char** argv) {
  const struct {
    const char* name;
    void (*run)();
  } all[] = {{"idle_after_frees", idle_after_frees},
             {"give_back", give_back},
             {"large_gets_the_rest", large_gets_the_rest},
             {"lasting_and_small", lasting_and_small},
             {"other_device", other_device},
             {"refused_free", refused_free},
             {"shared_buffers", shared_buffers}};
  for (const auto& t : all)
    if (!strcmp(argv[1], t.name)) return t.run(), 0;
  return 2;
}
