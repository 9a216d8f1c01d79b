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
#include <cuda_runtime.h>

#include <algorithm>
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
std::vector<Pinned> g_pinned;  // idle
int64_t g_holders = 0;

cudaMemPool_t device_pool() {
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
  }
  return g_pool[dev];
}

}  // namespace

void* ws_alloc(size_t bytes, cudaStream_t st) {
  if (!bytes) return nullptr;
  void* p = nullptr;
  cudaMemPool_t pool = device_pool();
  if (cudaMallocFromPoolAsync(&p, bytes, pool, st) != cudaSuccess) {
    cudaGetLastError();
    ws_trim();
    MB_CUDA(cudaMallocFromPoolAsync(&p, bytes, pool, st));
  }
  return p;
}

void ws_free(void* p, cudaStream_t st) {
  if (p) cudaFreeAsync(p, st);
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
  cudaDeviceSynchronize();
  std::lock_guard<std::mutex> lk(g_mu);
  for (cudaMemPool_t pool : g_pool)
    if (pool) cudaMemPoolTrimTo(pool, 0);
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
