// device_pool.h -- the library's work memory: a stream-ordered pool per device
// for buffers that live inside one call (tree builds, scene uploads).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace kdgr {

// Bytes a device's pool keeps mapped while no call uses it.  Mapping and
// unmapping a small build's buffers took longer than its kernels (creating a
// pool, mapping 1 MB and destroying it: 1.5 ms; an allocation from a pool
// that has the memory: 1 us).
constexpr size_t kWorkPoolKeep = 256ull << 20;

// Enter a call that takes work memory on device `dev` (the current device):
// the pool keeps everything it has mapped until the last such call leaves,
// then trims to kWorkPoolKeep.  Allocations and releases are stream-ordered,
// so calls on several threads and streams may share the pool.
cudaError_t work_pool_enter(int dev, cudaMemPool_t* out);
void work_pool_leave(int dev);
// Hand back what the pool of `dev` keeps (kdgr_shutdown).
void work_pool_trim(int dev);

}  // namespace kdgr
