// failures.cpp -- host-side failures on purpose, against the library's objects
// linked into this program: one `new` that throws, one CUDA runtime call that a
// wrapper (ld --wrap) answers with an error or a small number.  No failure
// reaches a kernel.  Usage: failures <case>; exit code 0 when it holds.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstdint>
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
// device memory, counted: from the host for cases that launch nothing, or from
// a device that says it has no more than g_capacity bytes
static bool g_fake_memory = false;
static long g_blocks = 0;
static size_t g_capacity = SIZE_MAX, g_taken = 0, g_free_reported = 0;
static struct {
  void* p;
  size_t n;
} g_sizes[64];  // the blocks handed out (no container: its own new would be counted)
static void note_block(void* key, void* p, size_t n) {
  for (auto& b : g_sizes)
    if (b.p == key) {
      g_taken += n - b.n;
      b = {p, n};
      return;
    }
}
cudaError_t __real_cudaMalloc(void** p, size_t n);
cudaError_t __wrap_cudaMalloc(void** p, size_t n) {
  if (!g_fake_memory) {
    if (n > g_capacity - g_taken) return cudaErrorMemoryAllocation;
    const cudaError_t e = __real_cudaMalloc(p, n);
    if (e == cudaSuccess) {
      ++g_blocks;
      note_block(nullptr, *p, n);
    }
    return e;
  }
  ++g_blocks;
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t __real_cudaFree(void* p);
cudaError_t __wrap_cudaFree(void* p) {
  if (p) --g_blocks;
  if (!g_fake_memory) {
    if (p) note_block(p, nullptr, 0);
    return __real_cudaFree(p);
  }
  std::free(p);
  return cudaSuccess;
}
cudaError_t __real_cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k);
cudaError_t __wrap_cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  if (!g_fake_memory) return __real_cudaMemcpy(d, s, n, k);
  std::memcpy(d, s, n);
  return cudaSuccess;
}
// stand-ins for memory pools on devices that this machine need not have
struct FakePool {
  int dev;
  size_t mapped;  // what the pool holds of its device
};
static bool g_fake_pools = false;
static int g_device = 0;
static std::vector<FakePool*> g_pools;
cudaError_t __real_cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps* props);
cudaError_t __wrap_cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps* props) {
  if (!g_fake_pools) return __real_cudaMemPoolCreate(p, props);
  FakePool* f = new FakePool{props->location.id, 1u << 20};
  g_pools.push_back(f);
  *p = reinterpret_cast<cudaMemPool_t>(f);
  return cudaSuccess;
}
cudaError_t __real_cudaMemPoolSetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void* v);
cudaError_t __wrap_cudaMemPoolSetAttribute(cudaMemPool_t p, cudaMemPoolAttr a, void* v) {
  return g_fake_pools ? cudaSuccess : __real_cudaMemPoolSetAttribute(p, a, v);
}
cudaError_t __real_cudaMemPoolTrimTo(cudaMemPool_t p, size_t keep);
cudaError_t __wrap_cudaMemPoolTrimTo(cudaMemPool_t p, size_t keep) {
  if (!g_fake_pools) return __real_cudaMemPoolTrimTo(p, keep);
  FakePool* f = reinterpret_cast<FakePool*>(p);
  if (f->mapped > keep) f->mapped = keep;
  return cudaSuccess;
}
cudaError_t __real_cudaMemPoolDestroy(cudaMemPool_t p);
cudaError_t __wrap_cudaMemPoolDestroy(cudaMemPool_t p) {
  if (!g_fake_pools) return __real_cudaMemPoolDestroy(p);
  reinterpret_cast<FakePool*>(p)->mapped = 0;
  return cudaSuccess;
}
cudaError_t __real_cudaMemGetInfo(size_t* free_bytes, size_t* total);
cudaError_t __wrap_cudaMemGetInfo(size_t* free_bytes, size_t* total) {
  if (!g_fake_pools) {
    const cudaError_t e = __real_cudaMemGetInfo(free_bytes, total);
    if (g_free_reported) *free_bytes = g_free_reported;
    return e;
  }
  *free_bytes = *total = size_t(1) << 32;
  return cudaSuccess;
}
cudaError_t __real_cudaGetDevice(int* dev);
cudaError_t __wrap_cudaGetDevice(int* dev) {
  if (!g_fake_pools) return __real_cudaGetDevice(dev);
  *dev = g_device;
  return cudaSuccess;
}
cudaError_t __real_cudaDeviceSynchronize();
cudaError_t __wrap_cudaDeviceSynchronize() { return g_fake_pools ? cudaSuccess : __real_cudaDeviceSynchronize(); }
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

// Every `new` of a scene's creation, in all forms, fails once.
static int scene_alloc() {
  const uint32_t n = 3000;
  std::vector<float> g = records(n);
  for (uint32_t i = 0; i < n; i += 16) g[64ull * i + 4] = 1e-6f;  // flagged in the packed form
  kdgr_tree t;
  REQUIRE(kdgr_init(0) == KDGR_OK);
  REQUIRE(kdgr_build_tree(g.data(), n, nullptr, &t, nullptr) == KDGR_OK);
  const long blocks = g_blocks, pool_blocks = g_pool_blocks;
  int failed = 0;
  for (long k = 0;; ++k) {
    kdgr_scene_t scene = nullptr;
    int rc = -1;
    g_new_left = k;
    try {
      rc = kdgr_scene_create(t.nodes, t.n_nodes, t.offsets, t.n_offsets, t.aabb, g.data(), n,
                             KDGR_FORM_EXACT | KDGR_FORM_FAST | KDGR_FORM_PACKED, &scene);
    } catch (...) {
      rc = -2;
    }
    const bool fired = g_new_left.exchange(-1) < 0;
    REQUIRE(rc != -2);  // an exception left the C entry
    REQUIRE(rc == (fired ? KDGR_ERR_OUT_OF_MEMORY : KDGR_OK));
    failed += fired;
    if (rc == KDGR_OK) REQUIRE(kdgr_scene_destroy(scene) == KDGR_OK);
    REQUIRE(g_blocks == blocks && g_pool_blocks == pool_blocks);
    if (!fired) break;
  }
  REQUIRE(failed > 10);
  REQUIRE(kdgr_shutdown() == KDGR_OK);
  uint64_t reserved = 1;
  REQUIRE(pool_reserved(&reserved) == 0);
  REQUIRE(reserved == 0);
  kdgr_tree_free(&t);
  return 0;
}

// One 96x64 frame of the plain form.
static int frame(kdgr_scene_t scene, std::vector<float>& out) {
  const kdgr_camera cam = {{0.f, 0.f, 1.6f}, {1.f, 0.f, 0.f}, {0.f, 1.f, 0.f}, {0.f, 0.f, 1.f}, 50.0, 1.5, 0.01};
  float* d = nullptr;
  out.assign(96 * 64 * 3, -1.f);
  REQUIRE(cudaMalloc(&d, out.size() * 4) == cudaSuccess);
  REQUIRE(kdgr_render(scene, &cam, 96, 64, d, nullptr, nullptr, nullptr, nullptr) == KDGR_OK);
  REQUIRE(cudaMemcpy(out.data(), d, out.size() * 4, cudaMemcpyDeviceToHost) == cudaSuccess);
  REQUIRE(cudaFree(d) == cudaSuccess);
  return 0;
}

static int scene_bytes(const kdgr_tree& t, const std::vector<float>& g, uint32_t forms, uint64_t* bytes,
                       std::vector<float>* img) {
  kdgr_scene_t s = nullptr;
  REQUIRE(kdgr_scene_create(t.nodes, t.n_nodes, t.offsets, t.n_offsets, t.aabb, g.data(), (uint32_t)(g.size() / 64),
                            forms, &s) == KDGR_OK);
  kdgr_scene_info i;
  REQUIRE(kdgr_scene_info_get(s, &i) == KDGR_OK);
  *bytes = i.device_bytes;
  if (img && (forms & KDGR_FORM_EXACT) && frame(s, *img)) return 1;
  REQUIRE(kdgr_scene_destroy(s) == KDGR_OK);
  return 0;
}

// On a device with room for what a scene's forms cannot do without, the scene
// is made whatever part of the plain form's leaf order would fit too.
static int scene_room() {
  const uint32_t n = 4000;
  const std::vector<float> g = records(n);
  kdgr_tree t;
  REQUIRE(kdgr_init(0) == KDGR_OK);
  REQUIRE(kdgr_build_tree(g.data(), n, nullptr, &t, nullptr) == KDGR_OK);
  for (uint32_t other : {0u, KDGR_FORM_FAST, KDGR_FORM_PACKED, KDGR_FORM_FAST | KDGR_FORM_PACKED}) {
    uint64_t without = 8ull * t.n_nodes + 80ull * n, full = 0, bytes = 0;
    std::vector<float> want, got;
    if (other) {
      if (scene_bytes(t, g, other, &bytes, nullptr)) return 1;
      without += bytes;
    } else {
      without += 4ull * t.n_offsets + 192ull * n + 4;
    }
    if (scene_bytes(t, g, KDGR_FORM_EXACT | other, &full, &want)) return 1;
    const uint64_t besides = 256ull * n + 96 * 64 * 12 + 8192;  // records, frame, rounding of the arrays
    REQUIRE(full > without + 100000);
    for (int k = 0; k <= 8; ++k) {
      g_capacity = without + besides + (full - without) * k / 8;
      if (scene_bytes(t, g, KDGR_FORM_EXACT | other, &bytes, &got)) {
        std::fprintf(stderr, "forms %x, step %d: %zu of %zu..%zu bytes\n", other, k, g_capacity, (size_t)without, (size_t)full);
        return 1;
      }
      REQUIRE(bytes <= g_capacity && got == want);
      REQUIRE(k < 8 || bytes == full);
    }
    g_capacity = SIZE_MAX;
  }
  kdgr_tree_free(&t);
  return 0;
}

// A large leaf order stays within an eighth of the free memory.
static int scene_share() {
  const uint32_t n = 20000;
  const std::vector<float> g = records(n);
  std::vector<float> want, got;
  kdgr_tree t;
  REQUIRE(kdgr_init(0) == KDGR_OK);
  REQUIRE(kdgr_build_tree_gpu(g.data(), n, nullptr, &t, nullptr) == KDGR_OK);
  uint64_t full = 0, bytes = 0;
  if (scene_bytes(t, g, KDGR_FORM_EXACT, &full, &want)) return 1;
  const uint64_t order = 60ull * t.n_offsets;  // at least
  REQUIRE(order > (100u << 20) && full > order);
  g_free_reported = 8 * order - 1;
  if (scene_bytes(t, g, KDGR_FORM_EXACT, &bytes, &got)) return 1;
  REQUIRE(bytes < full - order && got == want);
  g_free_reported = 12 * order;
  if (scene_bytes(t, g, KDGR_FORM_EXACT, &bytes, &got)) return 1;
  REQUIRE(bytes == full && got == want);
  kdgr_tree_free(&t);
  return 0;
}

// kdgr_shutdown gives back every device's work pool, except one in use.
static int shutdown_pools() {
  g_fake_pools = true;
  cudaMemPool_t p = nullptr;
  for (int dev : {0, 1, 5}) REQUIRE(kdgr::work_pool_enter(dev, &p) == cudaSuccess);
  kdgr::work_pool_leave(0);
  kdgr::work_pool_leave(1);
  REQUIRE(g_pools.size() == 3);
  REQUIRE(kdgr_shutdown() == KDGR_OK);
  REQUIRE(g_pools[0]->mapped == 0 && g_pools[1]->mapped == 0 && g_pools[2]->mapped > 0);
  kdgr::work_pool_leave(5);
  g_device = 1;
  REQUIRE(kdgr_shutdown() == KDGR_OK);
  for (const FakePool* f : g_pools) REQUIRE(f->mapped == 0);
  REQUIRE(kdgr::work_pool_enter(1, &p) == cudaSuccess);
  kdgr::work_pool_leave(1);
  return 0;
}

// Every `new` of a secondary scene's creation fails once.
static int secondary_alloc() {
  g_fake_memory = true;
  std::vector<float> tris(9 * 700);
  for (size_t i = 0; i < tris.size(); ++i) tris[i] = (float)(i % 11) * 0.1f + (float)(i % 9 == 4);
  kdgr_sphere sp[2];
  REQUIRE(kdgr_demo_spheres(sp) == KDGR_OK);
  int failed = 0;
  for (long k = 0;; ++k) {
    kdgr_secondary_t sec = nullptr;
    int rc = -1;
    g_new_left = k;
    try {
      rc = kdgr_secondary_create(sp, 2, tris.data(), 700, &sp[0].material, &sec);
    } catch (...) {
      rc = -2;
    }
    const bool fired = g_new_left.exchange(-1) < 0;
    REQUIRE(rc != -2);  // an exception left the C entry
    REQUIRE(rc == (fired ? KDGR_ERR_OUT_OF_MEMORY : KDGR_OK));
    failed += fired;
    if (rc == KDGR_OK) REQUIRE(kdgr_secondary_destroy(sec) == KDGR_OK);
    REQUIRE(g_blocks == 0);
    if (!fired) break;
  }
  REQUIRE(failed >= 3);
  return 0;
}

int main(int argc, char** argv) {
  const char* c = argc > 1 ? argv[1] : "";
  if (!std::strcmp(c, "build_alloc")) return build_alloc(2000);
  if (!std::strcmp(c, "build_alloc_threads")) return build_alloc(70000);  // four host ranges
  if (!std::strcmp(c, "shutdown_pools")) return shutdown_pools();
  if (!std::strcmp(c, "secondary_alloc")) return secondary_alloc();
  if (!std::strcmp(c, "scene_alloc")) return scene_alloc();
  if (!std::strcmp(c, "scene_room")) return scene_room();
  if (!std::strcmp(c, "scene_share")) return scene_share();
  std::fprintf(stderr, "unknown case %s\n", c);
  return 2;
}
