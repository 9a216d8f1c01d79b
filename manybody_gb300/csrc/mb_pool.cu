// Workspaces of the solvers: stream-ordered device memory and page-locked host
// buffers that are kept between calls.
//
// A solver call needs half a dozen vectors, its kept Lanczos vectors and a
// page-locked buffer for its scalars.  cudaMalloc and cudaFree cost 75 us a pair
// and 0.75 ms a GB (mapping), cudaMallocHost about 150 us: a 50-step solve of a
// 63,504-state sector spent 1.2 of its 2.1 ms on them.  Here each device has one
// CUDA memory pool that keeps up to 1/32 of the device's memory mapped for the
// next call; more is given back as soon as it is free, everything when the last
// operator and engine of the process are destroyed, and what is idle whenever
// an allocation does not fit otherwise.  A block is freed in the order of the
// stream it was used on; CUDA's pools serve any thread and stream.
//
// A block that would take the pool past what it keeps is cudaMalloc's: it could
// not be kept, and the pool maps and unmaps memory more slowly than cudaMalloc
// and cudaFree do.  From the second call on: a complex64 ground state of 1D L=16
// 8+8 (U = 2, 100 steps, 132 GB of kept Lanczos vectors) 0.71 -> 0.54 s, 4x4 6+6, 40
// steps, 167 -> 143 ms (151 with a line at twice what is kept), Q64, 20 steps, 149
// -> 106, complex64 4x4 5+5, 40 steps, 39.3 -> 38.1.
#include <cuda_runtime.h>

#include <algorithm>
#include <unordered_set>
#include <vector>

#include "mb_internal.h"

namespace mb {
namespace {

constexpr int kPoolDevices = 64;
constexpr size_t kPinnedUnit = size_t(64) << 10;
constexpr size_t kPinnedKeep = size_t(2) << 20;  // page-locked bytes kept idle at most

struct Pinned {
  void* p;
  size_t bytes;
};

std::mutex g_mu;
cudaMemPool_t g_pool[kPoolDevices] = {};
uint64_t g_keep[kPoolDevices] = {};        // bytes kept mapped
std::unordered_set<void*> g_apart;         // blocks of cudaMalloc
std::vector<Pinned> g_pinned;  // idle
int64_t g_holders = 0;

cudaMemPool_t device_pool(uint64_t* keep_out = nullptr) {
  int dev = 0;
  MB_CUDA(cudaGetDevice(&dev));
  MB_REQUIRE(dev >= 0 && dev < kPoolDevices, MB_ERR_CAPACITY, "device ordinal above 63");
  std::lock_guard<std::mutex> lk(g_mu);
  if (!g_pool[dev]) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    MB_CUDA(cudaMemPoolCreate(&pool, &props));
    size_t free_b = 0, total_b = 0;
    MB_CUDA(cudaMemGetInfo(&free_b, &total_b));
    uint64_t keep = total_b / 32;
    MB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    g_pool[dev] = pool;
    g_keep[dev] = keep;
  }
  if (keep_out) *keep_out = g_keep[dev];
  return g_pool[dev];
}

constexpr size_t kLargeBlock = size_t(64) << 20;  // smaller ones are the pool's without a look

// Whether a block would take the pool past what it keeps.
bool too_large(cudaMemPool_t pool, size_t bytes, uint64_t keep) {
  uint64_t used = 0;
  if (bytes < kLargeBlock) return false;
  MB_CUDA(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used));
  return used + bytes > keep;
}

}  // namespace

void* ws_alloc(size_t bytes, cudaStream_t st) {
  if (!bytes) return nullptr;
  void* p = nullptr;
  uint64_t keep = 0;
  cudaMemPool_t pool = device_pool(&keep);
  if (too_large(pool, bytes, keep)) {
    MB_CUDA(dev_malloc(&p, bytes));
    std::lock_guard<std::mutex> lk(g_mu);
    g_apart.insert(p);
    return p;
  }
  if (cudaMallocFromPoolAsync(&p, bytes, pool, st) != cudaSuccess) {
    cudaGetLastError();
    ws_trim();
    MB_CUDA(cudaMallocFromPoolAsync(&p, bytes, pool, st));
  }
  return p;
}

void ws_free(void* p, cudaStream_t st) {
  if (!p) return;
  bool apart;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    apart = g_apart.erase(p) > 0;
  }
  if (apart) cudaFree(p);
  else cudaFreeAsync(p, st);
}

size_t ws_idle() {
  uint64_t reserved = 0, used = 0;
  int dev = 0;
  MB_CUDA(cudaGetDevice(&dev));
  cudaMemPool_t pool = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (dev >= 0 && dev < kPoolDevices) pool = g_pool[dev];
  }
  if (!pool) return 0;  // not made for the question
  if (cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &reserved) != cudaSuccess ||
      cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return reserved > used ? (size_t)(reserved - used) : 0;
}

void ws_trim() {
  cudaMemPool_t pools[kPoolDevices];
  {
    std::lock_guard<std::mutex> lk(g_mu);
    std::copy(g_pool, g_pool + kPoolDevices, pools);
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return;
  for (int d = 0; d < kPoolDevices; ++d)
    if (pools[d] && cudaSetDevice(d) == cudaSuccess) {
      cudaDeviceSynchronize();  // blocks freed in the order of a stream are back
      cudaMemPoolTrimTo(pools[d], 0);
    }
  cudaSetDevice(dev);
}

cudaError_t dev_malloc(void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation && ws_idle() > 0) {
    cudaGetLastError();
    ws_trim();
    e = cudaMalloc(p, bytes);
  }
  return e;
}

void* pinned_take(size_t bytes) {
  const size_t size = std::max<size_t>((bytes + kPinnedUnit - 1) / kPinnedUnit, 1) * kPinnedUnit;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    for (size_t i = 0; i < g_pinned.size(); ++i)
      if (g_pinned[i].bytes == size) {
        void* p = g_pinned[i].p;
        g_pinned.erase(g_pinned.begin() + (std::ptrdiff_t)i);
        return p;
      }
  }
  void* p = nullptr;
  MB_CUDA(cudaMallocHost(&p, size));
  return p;
}

void pinned_give(void* p, size_t bytes) {
  if (!p) return;
  const size_t size = std::max<size_t>((bytes + kPinnedUnit - 1) / kPinnedUnit, 1) * kPinnedUnit;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    size_t idle = size;
    for (const Pinned& b : g_pinned) idle += b.bytes;
    if (g_holders > 0 && idle <= kPinnedKeep) {
      g_pinned.push_back({p, size});
      return;
    }
  }
  cudaFreeHost(p);
}

void ws_hold() {
  std::lock_guard<std::mutex> lk(g_mu);
  ++g_holders;
}

void ws_drop() {
  std::vector<Pinned> idle;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (--g_holders > 0) return;
    idle.swap(g_pinned);
  }
  for (const Pinned& b : idle) cudaFreeHost(b.p);
  ws_trim();
}

}  // namespace mb
