// device_pool.cpp -- see device_pool.h.
#include "device_pool.h"

#include <cstdint>
#include <mutex>

namespace kdgr {
namespace {
constexpr int kMaxDevices = 64;
struct Pools {
  std::mutex mu;
  cudaMemPool_t pool[kMaxDevices] = {};
  int users[kMaxDevices] = {};
  size_t keep[kMaxDevices] = {};
};
Pools& pools() {
  static Pools p;
  return p;
}
}  // namespace

cudaError_t work_pool_enter(int dev, cudaMemPool_t* out) {
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  Pools& P = pools();
  std::lock_guard<std::mutex> lk(P.mu);
  if (!P.pool[dev]) {
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    cudaMemPool_t pool = nullptr;
    cudaError_t e = cudaMemPoolCreate(&pool, &props);
    if (e != cudaSuccess) return e;
    uint64_t keep = UINT64_MAX;
    e = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) {
      cudaMemPoolDestroy(pool);
      return e;
    }
    size_t free_bytes = 0, total = 0;
    if (cudaMemGetInfo(&free_bytes, &total) != cudaSuccess) total = 0;
    P.keep[dev] = total / kWorkPoolShare;
    P.pool[dev] = pool;
  }
  ++P.users[dev];
  *out = P.pool[dev];
  return cudaSuccess;
}

void work_pool_leave(int dev) {
  if (dev < 0 || dev >= kMaxDevices) return;
  Pools& P = pools();
  std::lock_guard<std::mutex> lk(P.mu);
  if (--P.users[dev] == 0) cudaMemPoolTrimTo(P.pool[dev], P.keep[dev]);
}

cudaError_t work_pool_release() {
  Pools& P = pools();
  std::lock_guard<std::mutex> lk(P.mu);
  cudaError_t first = cudaSuccess;
  for (int dev = 0; dev < kMaxDevices; ++dev) {
    if (!P.pool[dev] || P.users[dev] != 0) continue;
    const cudaError_t e = cudaMemPoolDestroy(P.pool[dev]);
    if (first == cudaSuccess) first = e;
    P.pool[dev] = nullptr;
  }
  return first;
}

}  // namespace kdgr
