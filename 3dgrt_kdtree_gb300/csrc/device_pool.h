// device_pool.h -- the library's work memory: a stream-ordered pool per device
// for buffers that live inside one call (tree builds, scene uploads).
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace kdgr {

// A device's pool keeps up to 1/64 of the device's memory mapped while no call
// uses it (4.3 of 277 GiB on a GB300).  Mapping and unmapping a small build's
// buffers took longer than its kernels (creating a pool, mapping 1 MB and
// destroying it: 1.5 ms; an allocation from a pool that has the memory: 1 us),
// and a 500k-Gaussian build's 3 GB took 5 of its 75 ms.
constexpr size_t kWorkPoolShare = 64;

// Enter a call that takes work memory on device `dev` (the current device):
// the pool keeps everything it has mapped until the last such call leaves,
// then trims to its share.  Allocations and releases are stream-ordered,
// so calls on several threads and streams may share the pool.
cudaError_t work_pool_enter(int dev, cudaMemPool_t* out);
void work_pool_leave(int dev);
// Hand back the pools that no call is in, on every device (kdgr_shutdown); the
// next call on a device makes a new one.
cudaError_t work_pool_release();

}  // namespace kdgr
