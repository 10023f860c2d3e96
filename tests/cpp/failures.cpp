// failures.cpp -- host-side failures on purpose, against the library's objects
// linked into this program: one `new` that throws, one CUDA runtime call that a
// wrapper (ld --wrap) answers with an error or a small number.  No failure
// reaches a kernel.  Usage: failures <case>; exit code 0 when it holds.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>
#include <vector>

#include "device_pool.h"
#include "kdgr.h"

// ------------------------------------------------------------ one throwing new
static std::atomic<long> g_new_left{-1};  // new calls until one throws; < 0: none does
void* operator new(std::size_t n) {
  if (g_new_left.load() >= 0 && g_new_left.fetch_sub(1) == 0) throw std::bad_alloc();
  void* p = std::malloc(n ? n : 1);
  if (!p) throw std::bad_alloc();
  return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

// ------------------------------------------------------------ wrapped calls
static long g_streams = 0, g_pool_blocks = 0;
extern "C" {
cudaError_t __real_cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f);
cudaError_t __wrap_cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) {
  const cudaError_t e = __real_cudaStreamCreateWithFlags(s, f);
  if (e == cudaSuccess) ++g_streams;
  return e;
}
cudaError_t __real_cudaStreamDestroy(cudaStream_t s);
cudaError_t __wrap_cudaStreamDestroy(cudaStream_t s) {
  --g_streams;
  return __real_cudaStreamDestroy(s);
}
cudaError_t __real_cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t s);
cudaError_t __wrap_cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t pool, cudaStream_t s) {
  const cudaError_t e = __real_cudaMallocFromPoolAsync(p, n, pool, s);
  if (e == cudaSuccess) ++g_pool_blocks;
  return e;
}
cudaError_t __real_cudaFreeAsync(void* p, cudaStream_t s);
cudaError_t __wrap_cudaFreeAsync(void* p, cudaStream_t s) {
  --g_pool_blocks;
  return __real_cudaFreeAsync(p, s);
}
}

#define REQUIRE(c)                                                      \
  do {                                                                  \
    if (!(c)) {                                                         \
      std::fprintf(stderr, "line %d: %s (last error: %s)\n", __LINE__, #c, kdgr_last_error()); \
      return 1;                                                         \
    }                                                                   \
  } while (0)

// Gaussians of a small cube, spread by a fixed sequence.
static std::vector<float> records(uint32_t n) {
  std::vector<float> g(64ull * n, 0.f);
  uint32_t x = 1;
  auto u = [&] { return (float)((x = x * 1664525u + 1013904223u) >> 8) / 16777216.f; };
  for (uint32_t i = 0; i < n; ++i) {
    float* r = &g[64ull * i];
    for (int d = 0; d < 3; ++d) r[d] = u() - 0.5f;
    r[3] = 0.2f + 0.7f * u();
    for (int d = 0; d < 3; ++d) r[4 + d] = 0.01f + 0.02f * u();
    r[7] = 1.f;
    r[8] = 1.f;
    for (int d = 12; d < 60; ++d) r[d] = 0.3f * u();
  }
  return g;
}

// What the work pool of device 0 has mapped once nothing uses it.
static int pool_reserved(uint64_t* out) {
  cudaMemPool_t pool = nullptr;
  if (kdgr::work_pool_enter(0, &pool) != cudaSuccess) return 1;
  const cudaError_t e = cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, out);
  kdgr::work_pool_leave(0);
  return e != cudaSuccess;
}

// Every `new` of a device build fails once: the call says so, leaves the
// caller's tree alone, and gives back its stream, buffers and pool entry.
static int build_alloc(uint32_t n) {
  const std::vector<float> g = records(n);
  kdgr_tree t;
  REQUIRE(kdgr_init(0) == KDGR_OK);
  REQUIRE(kdgr_build_tree_gpu(g.data(), n, nullptr, &t, nullptr) == KDGR_OK);
  kdgr_tree_free(&t);
  const long streams = g_streams, blocks = g_pool_blocks;
  int failed = 0;
  for (long k = 0;; ++k) {
    g_new_left = k;
    const int rc = kdgr_build_tree_gpu(g.data(), n, nullptr, &t, nullptr);
    const bool fired = g_new_left.exchange(-1) < 0;
    REQUIRE(rc == KDGR_OK || (fired && rc == KDGR_ERR_OUT_OF_MEMORY));
    if (rc == KDGR_OK) kdgr_tree_free(&t);
    else ++failed;
    REQUIRE(g_streams == streams && g_pool_blocks == blocks);
    if (!fired) break;
  }
  REQUIRE(failed > 5);
  REQUIRE(kdgr_shutdown() == KDGR_OK);
  uint64_t reserved = 1;
  REQUIRE(pool_reserved(&reserved) == 0);
  REQUIRE(reserved == 0);
  return 0;
}

int main(int argc, char** argv) {
  const char* c = argc > 1 ? argv[1] : "";
  if (!std::strcmp(c, "build_alloc")) return build_alloc(2000);
  if (!std::strcmp(c, "build_alloc_threads")) return build_alloc(70000);  // four host ranges
  std::fprintf(stderr, "unknown case %s\n", c);
  return 2;
}
