// device_memory.cpp — see device_memory.cuh.
#include "device_memory.cuh"

#include <cstdint>
#include <map>
#include <mutex>

namespace gwmb {
namespace {

constexpr uint64_t kKeptScratch = 256ull << 20;
std::mutex pools_lock;
std::map<int, cudaMemPool_t> pools;

// The device's pool, made at its first use; null where it cannot be had.
cudaMemPool_t pool_of(int dev) {
  std::lock_guard<std::mutex> hold(pools_lock);
  const auto it = pools.find(dev);
  if (it != pools.end()) return it->second;
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = dev;
  cudaMemPool_t pool = nullptr;
  if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
    cudaGetLastError();
    return nullptr;
  }
  uint64_t keep = kKeptScratch;
  if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
    cudaMemPoolDestroy(pool);
    cudaGetLastError();
    return nullptr;
  }
  pools[dev] = pool;
  return pool;
}

template <class Try>
cudaError_t with_retry(Try&& attempt) {
  cudaError_t e = attempt();
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  trim_scratch();
  e = attempt();
  if (e == cudaErrorMemoryAllocation) cudaGetLastError();
  return e;
}

}  // namespace

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
  int dev = 0;
  const cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (const cudaMemPool_t pool = pool_of(dev)) {
    const cudaError_t a = with_retry([&] { return cudaMallocFromPoolAsync(p, bytes, pool, s); });
    if (a == cudaSuccess || a == cudaErrorMemoryAllocation) return a;
    cudaGetLastError();  // a pool of a context that is gone (cudaDeviceReset): forget it
    std::lock_guard<std::mutex> hold(pools_lock);
    const auto it = pools.find(dev);
    if (it != pools.end() && it->second == pool) pools.erase(it);
  }
  return device_alloc_async_bytes(p, bytes, s);
}

void trim_scratch() {
  std::lock_guard<std::mutex> hold(pools_lock);
  for (const auto& [dev, pool] : pools)
    if (cudaMemPoolTrimTo(pool, 0) != cudaSuccess) cudaGetLastError();
}

cudaError_t device_alloc_bytes(void** p, size_t bytes) {
  return with_retry([&] { return cudaMalloc(p, bytes); });
}
cudaError_t device_alloc_async_bytes(void** p, size_t bytes, cudaStream_t s) {
  return with_retry([&] { return cudaMallocAsync(p, bytes, s); });
}

}  // namespace gwmb
