// kdgr_api.cpp -- C ABI: device selection, scene upload, plain render calls.
//
// Scene upload replaces renderGaussianWithCudaSetup (cudaRenderer.cu:
// 2557-2703): where the reference copies the tree and the 256-byte AoS
// Gaussians once and binds texture objects (then destroys them, :2693-2702),
// this validates the tree, builds the device layouts each render form reads
// (see device_common.cuh) and keeps them for the scene's lifetime.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <deque>
#include <memory>
#include <string>
#include <vector>

#include "kdgr_internal.h"
#include "scene.h"

namespace kdgr {

int cuda_fail(cudaError_t e, const char* where) {
  set_error(std::string(where) + ": " + cudaGetErrorString(e));
  cudaGetLastError();  // clear a sticky launch-configuration error
  return e == cudaErrorMemoryAllocation ? KDGR_ERR_OUT_OF_MEMORY : KDGR_ERR_CUDA;
}

CamInfo make_caminfo(const kdgr_camera& cam, int width, int height) {
  CamInfo c;
  const float kPi = 3.14159265358979323846f;  // M_PI as cudaRenderer.h:31 defines it
  const float fov_rad = (float)(cam.fovy * (kPi / 180.0f));
  const float plane_height = (float)(2.0f * cam.near_c * tanf(fov_rad * 0.5f));
  const float plane_width = (float)(plane_height * cam.aspect);
  c.step_x = plane_width / width;
  c.step_y = plane_height / height;
  const float nc = (float)cam.near_c;
  for (int i = 0; i < 3; ++i) {
    c.eye[i] = cam.pos[i];
    c.u[i] = cam.uaxis[i];
    c.v[i] = cam.vaxis[i];
    const float a = cam.pos[i] - cam.naxis[i] * nc;
    const float b = a - cam.uaxis[i] * (plane_width * 0.5f);
    c.start[i] = b + cam.vaxis[i] * (plane_height * 0.5f);
  }
  return c;
}

}  // namespace kdgr

using namespace kdgr;

kdgr::ExactView kdgr_scene_s::exact_view() const {
  ExactView v;
  v.nodes = d_nodes;
  v.offsets = d_offsets;
  v.test = d_test;
  v.sh = d_sh;
  v.n_nodes = n_nodes;
  v.n_offsets = n_offsets;
  v.n_gauss = n_gauss;
  for (int i = 0; i < 3; ++i) {
    v.bmin[i] = aabb[i];
    v.bmax[i] = aabb[3 + i];
  }
  return v;
}

kdgr::FastView kdgr_scene_s::fast_view(bool packed) const {
  FastView v;
  v.nodes = packed ? d_nodes_packed : d_nodes_fast;
  v.offsets = packed ? d_gid_plain : d_pair_gid;
  v.opacity = d_opacity;
  v.sh = d_sh;
  v.sh_bf16 = d_sh_bf16;
  v.leaf_pairs = packed ? d_flag_pairs : d_leaf_pairs;
  v.leaf_packed = d_leaf_packed;
  v.leaf_aux = packed ? d_leaf_aux : nullptr;
  v.flag_offsets = packed ? d_gid_flag : nullptr;
  v.n_nodes = n_nodes;
  v.n_offsets = packed ? n_plain_entries : n_pair_entries;
  v.n_flag = packed ? n_flag_entries : 0u;
  v.n_gauss = n_gauss;
  v.top_nodes = top_nodes;
  for (int i = 0; i < 3; ++i) {
    v.bmin[i] = aabb[i];
    v.bmax[i] = aabb[3 + i];
  }
  return v;
}

kdgr::PlainView kdgr_scene_s::plain_view() const {
  PlainView v;
  v.nodes = d_nodes_fast;
  v.offsets = d_pair_gid;
  v.leaf_pairs = d_leaf_pairs;
  v.leaf_tol = d_leaf_tol;
  v.leaf_first = d_leaf_first;
  v.test = d_test;
  v.sh = d_sh;
  v.n_offsets = n_pair_entries;
  v.n_gauss = n_gauss;
  for (int i = 0; i < 3; ++i) {
    v.bmin[i] = aabb[i];
    v.bmax[i] = aabb[3 + i];
  }
  return v;
}

namespace kdgr {

// Whether the plain form's leaf order may take `bytes` of the current device:
// above 64 MB at most an eighth of what is free, so that a scene does not fill
// the device with arrays that it can render without (the 1M cluster scene:
// 0.37 GB without them, 1.9 with).
static bool plain_order_fits(size_t bytes) {
  if (bytes <= (64u << 20)) return true;
  size_t free_bytes = 0, total = 0;
  return cudaMemGetInfo(&free_bytes, &total) == cudaSuccess && bytes <= free_bytes / 8;
}

// renderGaussianWithCudaSetup (cudaRenderer.cu:2557-2703) from device-resident
// 64-float records: the tree is copied to the device as given, checked,
// relaid out and expanded into padded leaf order there (scene_tree.cu), and
// the per-Gaussian arrays of every requested form are written by the packing
// kernel (scene_pack.cu).  Work runs on the legacy default stream, so that
// records another blocking stream is still writing are waited for.
int scene_create_impl(const uint32_t* nodes, uint32_t n_nodes, const uint32_t* offsets, uint32_t n_offsets,
                      const float aabb[6], uint32_t n, uint32_t flags,
                      const std::function<int(const float** d_gaussians)>& records, kdgr_scene_t* out,
                      const char* who) {
  const std::string w(who);
  uint32_t forms = flags & (KDGR_FORM_EXACT | KDGR_FORM_FAST | KDGR_FORM_PACKED);
  if (forms == 0) forms = KDGR_FORM_EXACT | KDGR_FORM_FAST;
  const bool inverted = (flags & KDGR_SCALES_INVERTED) != 0;
  const bool exact = (forms & KDGR_FORM_EXACT) != 0, fast = (forms & KDGR_FORM_FAST) != 0,
             packed = (forms & KDGR_FORM_PACKED) != 0;

  struct Discard {  // a scene that is not handed out gives its arrays back
    void operator()(kdgr_scene_s* p) const {
      for (void* b : p->blocks) cudaFree(b);
      delete p;
    }
  };
  std::unique_ptr<kdgr_scene_s, Discard> s(new kdgr_scene_s);
  WorkMem W(nullptr);
  auto fail = [&](const char* where, cudaError_t e) {
    return cuda_fail(e != cudaSuccess ? e : cudaErrorUnknown, (w + ": " + where).c_str());
  };
  auto host_check = [&]() {  // names what is wrong with the tree
    std::string err;
    uint32_t depth = 0;
    const int rc = validate_tree(nodes, n_nodes, offsets, n_offsets, n, err, &depth);
    if (rc != KDGR_OK) set_error(w + ": " + err);
    return rc;
  };
  if (W.err != cudaSuccess) {  // a malformed tree is refused as such also without a device
    const int rc = host_check();
    return rc != KDGR_OK ? rc : fail("work memory", W.err);
  }
  s->device = W.dev;
  s->forms = forms;
  s->n_nodes = n_nodes;
  s->n_offsets = n_offsets;
  s->n_gauss = n;
  memcpy(s->aabb, aabb, sizeof(s->aabb));

  // the tree as given, and its checks
  uint2* d_raw = W.take<uint2>(n_nodes);
  uint32_t* d_ids = W.take<uint32_t>(n_offsets ? n_offsets : 1);
  cudaError_t e = W.err;
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_raw, nodes, 8ull * n_nodes, cudaMemcpyHostToDevice, W.st);
  if (e == cudaSuccess && n_offsets)
    e = cudaMemcpyAsync(d_ids, offsets, 4ull * n_offsets, cudaMemcpyHostToDevice, W.st);
  TreeLists L;
  if (e == cudaSuccess) e = tree_check(W, d_raw, n_nodes, d_ids, n_offsets, n, L);
  if (e != cudaSuccess) return fail("tree upload", e);
  if (!L.ok) {
    const int rc = host_check();
    if (rc != KDGR_OK) return rc;
    set_error(w + ": the tree failed its device check");
    return KDGR_ERR_FORMAT;
  }
  s->depth = L.levels - 1;
  s->n_leaves = L.n_leaves;
  s->max_leaf = L.max_leaf;
  const float* d_g = nullptr;
  const int rrc = records(&d_g);
  if (rrc != KDGR_OK) return rrc;

  Slab A;
  A.add(s->d_offsets, n_offsets ? n_offsets : 1);
  A.add(s->d_sh, 12 * (size_t)n);
  A.add(s->d_status, 1);
  if (exact) {
    A.add(s->d_nodes, n_nodes);
    A.add(s->d_test, kTestWords * (size_t)n);
  }
  if (fast || packed) A.add(s->d_nodes_fast, n_nodes);
  if (fast || packed) A.add(s->d_opacity, n);
  if (packed) {
    A.add(s->d_sh_bf16, 6 * (size_t)n);
    A.add(s->d_nodes_packed, n_nodes);
    A.add(s->d_leaf_aux, n_nodes);
  }
  e = A.make(s->blocks);
  if (e != cudaSuccess) return fail("cudaMalloc", e);
  if (n_offsets) e = cudaMemcpyAsync(s->d_offsets, d_ids, 4ull * n_offsets, cudaMemcpyDeviceToDevice, W.st);
  if (e == cudaSuccess && exact)
    e = cudaMemcpyAsync(s->d_nodes, d_raw, 8ull * n_nodes, cudaMemcpyDeviceToDevice, W.st);
  if (e == cudaSuccess) e = cudaMemsetAsync(s->d_status, 0, 4, W.st);
  if (e != cudaSuccess) return fail("tree arrays", e);

  // the relaid tree and its leaves' pairs
  uint2* const relaid = fast || packed ? s->d_nodes_fast : W.take<uint2>(n_nodes);
  uint64_t *first = nullptr, n_pairs = 0;
  e = W.err;
  if (e == cudaSuccess) e = tree_relayout(W, d_raw, L, relaid);
  if (e == cudaSuccess) e = tree_leaf_pairs(W, relaid, L.n, &first, &n_pairs);
  if (e != cudaSuccess) return fail("tree relayout", e);
  const bool fits = 2 * n_pairs <= 0xFFFFFFF0ull;
  if ((fast || packed) && !fits) {
    set_error(w + ": more than 2^32 leaf entries after pair padding");
    return KDGR_ERR_LIMIT;
  }
  if (fast || packed) s->top_nodes = L.top_nodes;

  // The plain form's leaf order only makes it faster: never at the cost of
  // what a form cannot do without, and within bounds.  It shares the last
  // allocation, as one of its own costs a scene its cudaFree (opening, drawing
  // and closing 115k / 180k overlapping Gaussians: 4.6 / 13.4 against 4.2 / 12.0 ms).
  auto add_plain = [&](Slab& X) {
    if (!(fast || packed)) {
      X.add(s->d_nodes_fast, n_nodes);
      X.add(s->d_pair_gid, 2 * n_pairs + 2);
    }
    if (!fast) X.add(s->d_leaf_pairs, 6 * (n_pairs + 1));
    X.add(s->d_leaf_tol, n_pairs + 1);
    X.add(s->d_leaf_first, n_nodes);
  };
  Slab X;
  if (exact) add_plain(X);
  bool plain = exact && fits && plain_order_fits(X.bytes);
  // `must` with the plain form's arrays when there is room for both, without otherwise
  auto make_last = [&](Slab& must) {
    if (plain) {
      Slab both = must;
      add_plain(both);
      if (both.make(s->blocks) == cudaSuccess) {
        must.bytes = both.bytes;
        return cudaSuccess;
      }
      cudaGetLastError();
      plain = false;
    }
    return must.at.empty() ? cudaSuccess : must.make(s->blocks);
  };

  // per-Gaussian arrays, packed on the device
  PackOut po{};
  po.sh = s->d_sh;
  po.test = s->d_test;
  po.opacity = s->d_opacity;
  po.sh_bf16 = s->d_sh_bf16;
  if (packed) po.giscl = W.take<float>(3 * (size_t)n);
  if (fast) po.fast = W.take<float4>(3 * (size_t)n);
  if (packed) po.packed = W.take<uint32_t>(8 * (size_t)n);
  if (packed) po.aniso = W.take<uint8_t>(n);
  if (W.err != cudaSuccess) return fail("cudaMalloc (staging)", W.err);
  if (plain && !fast) po.fast = W.try_take<float4>(3 * (size_t)n);
  if (plain) po.tol = W.try_take<float2>(n);
  plain = plain && po.fast && po.tol;
  e = launch_pack(d_g, n, inverted, po, W.st);
  if (e != cudaSuccess) return fail("packing kernel", e);

  // the fast forms' padded leaf order; the per-Gaussian rows are staging, the
  // kernels read the leaf-order pairs
  Slab P;
  if (fast || packed) {
    P.add(s->d_pair_gid, 2 * n_pairs + 2);
    if (fast) P.add(s->d_leaf_pairs, 6 * (n_pairs + 1));
    e = packed ? P.make(s->blocks) : make_last(P);
    if (e != cudaSuccess) return fail("cudaMalloc (leaf order)", e);
    s->n_pair_entries = (uint32_t)(2 * n_pairs);
    e = tree_leaf_gids(W, relaid, L.n, first, s->d_offsets, s->d_pair_gid);
    if (e == cudaSuccess && fast)
      e = build_leaf_pairs(s->d_pair_gid, s->n_pair_entries, po.fast, s->d_leaf_pairs, W.st);
    if (e != cudaSuccess) return fail("leaf order", e);
  }
  Slab Q;
  if (packed) {
    // the flagged Gaussians get FP64-precomputed factors, and each leaf is
    // laid out as its plain entries in FP16 pairs followed by its flagged
    // entries in FP32 pairs of a second stream
    uint32_t* aidx = nullptr;
    uint64_t *split = nullptr, totals = 0;
    e = aniso_index(W, po.aniso, n, &aidx, &s->n_aniso);
    if (e == cudaSuccess)
      e = tree_split_counts(W, s->d_nodes_fast, L.n, s->d_pair_gid, po.aniso, &split, &totals);
    if (e != cudaSuccess) return fail("packed leaf counts", e);
    s->n_plain_entries = 2u * (uint32_t)totals;
    s->n_flag_entries = 2u * (uint32_t)(totals >> 32);
    Q.add(s->d_gid_plain, s->n_plain_entries + 2ull);
    Q.add(s->d_gid_flag, s->n_flag_entries + 2ull);
    Q.add(s->d_leaf_packed, 2 * (s->n_plain_entries + 2ull));
    Q.add(s->d_flag_pairs, 3 * (s->n_flag_entries + 2ull));
    float* src = W.take<float>(10 * (size_t)s->n_aniso);
    float4* table = W.take<float4>(3 * (size_t)s->n_aniso);
    e = W.err;
    if (e == cudaSuccess) e = make_last(Q);
    if (e != cudaSuccess) return fail("cudaMalloc (packed)", e);
    e = tree_split_fill(W, s->d_nodes_fast, L.n, s->d_pair_gid, po.aniso, split, s->d_nodes_packed, s->d_leaf_aux,
                        s->d_gid_plain, s->d_gid_flag);
    if (e == cudaSuccess) e = build_packed_pairs(s->d_gid_plain, s->n_plain_entries, po.packed, s->d_leaf_packed, W.st);
    if (e == cudaSuccess && s->n_aniso) {
      e = launch_gather_aniso(d_g, po.giscl, aidx, n, src, W.st);
      if (e == cudaSuccess) e = launch_aniso_fp64(src, s->n_aniso, table, W.st);
      if (e == cudaSuccess) e = build_flag_pairs(s->d_gid_flag, s->n_flag_entries, aidx, table, s->d_flag_pairs, W.st);
    }
    if (e != cudaSuccess) return fail("packed upload", e);
  }
  // without room for its leaf order the plain form walks one thread per ray
  // over the tree as given
  if (!fast && !packed) make_last(P);
  if (plain) {
    e = cudaSuccess;
    if (!(fast || packed)) {
      s->n_pair_entries = (uint32_t)(2 * n_pairs);
      e = tree_leaf_gids(W, relaid, L.n, first, s->d_offsets, s->d_pair_gid);
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(s->d_nodes_fast, relaid, 8ull * L.n, cudaMemcpyDeviceToDevice, W.st);
    }
    if (e == cudaSuccess && !fast)
      e = build_leaf_pairs(s->d_pair_gid, s->n_pair_entries, po.fast, s->d_leaf_pairs, W.st);
    if (e == cudaSuccess) e = build_leaf_tol(s->d_pair_gid, s->n_pair_entries, po.tol, s->d_leaf_tol, W.st);
    if (e == cudaSuccess) e = tree_leaf_first(W, L, first, s->d_leaf_first);
    if (e != cudaSuccess) return fail("plain leaf order", e);
  }
  e = cudaStreamSynchronize(W.st);
  if (e != cudaSuccess) return fail("upload", e);
  s->device_bytes = A.bytes + P.bytes + Q.bytes;
  *out = s.release();
  return KDGR_OK;
}

}  // namespace kdgr

extern "C" {

int kdgr_init(int device) {
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return cuda_fail(e, "kdgr_init: cudaSetDevice");
  e = cudaFree(nullptr);
  if (e != cudaSuccess) return cuda_fail(e, "kdgr_init: context");
  return KDGR_OK;
}

int kdgr_shutdown(void) {
  cudaError_t e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = work_pool_release();
  if (e != cudaSuccess) return cuda_fail(e, "kdgr_shutdown");
  return KDGR_OK;
}

int kdgr_scene_create(const uint32_t* nodes, uint32_t n_nodes, const uint32_t* offsets, uint32_t n_offsets,
                      const float aabb[6], const float* g, uint32_t n, uint32_t flags, kdgr_scene_t* out) {
  if (!out || !nodes || !aabb || !g || n == 0 || n_nodes == 0 || (n_offsets && !offsets)) {
    set_error("kdgr_scene_create: null argument, no nodes or no Gaussians");
    return KDGR_ERR_INVALID_ARG;
  }
  *out = nullptr;
  // the records go to the device as they are; the device packs every form
  float* d_rec = nullptr;
  const int rc = host_guard("kdgr_scene_create", [&] {
    return scene_create_impl(
        nodes, n_nodes, offsets, n_offsets, aabb, n, flags,
        [&](const float** d) {
          cudaError_t e = cudaMalloc(&d_rec, 256ull * n);
          if (e == cudaSuccess) e = cudaMemcpyAsync(d_rec, g, 256ull * n, cudaMemcpyHostToDevice, nullptr);
          if (e != cudaSuccess) return cuda_fail(e, "kdgr_scene_create: record upload");
          *d = d_rec;
          return (int)KDGR_OK;
        },
        out, "kdgr_scene_create");
  });
  if (d_rec) cudaFree(d_rec);
  return rc;
}

int kdgr_scene_create_device(const uint32_t* nodes, uint32_t n_nodes, const uint32_t* offsets, uint32_t n_offsets,
                             const float aabb[6], const float* d_g, uint32_t n, uint32_t flags, kdgr_scene_t* out) {
  if (!out || !nodes || !aabb || !d_g || n == 0 || n_nodes == 0 || (n_offsets && !offsets)) {
    set_error("kdgr_scene_create_device: null argument, no nodes or no Gaussians");
    return KDGR_ERR_INVALID_ARG;
  }
  *out = nullptr;
  return host_guard("kdgr_scene_create_device", [&] {
    return scene_create_impl(
        nodes, n_nodes, offsets, n_offsets, aabb, n, flags,
        [&](const float** d) {
          *d = d_g;
          return (int)KDGR_OK;
        },
        out, "kdgr_scene_create_device");
  });
}

int kdgr_scene_destroy(kdgr_scene_t s) {
  if (!s) return KDGR_ERR_INVALID_ARG;
  DeviceScope on(s->device);
  cudaError_t first = cudaSuccess;
  for (void* p : s->blocks)
    if (p) {
      cudaError_t e = cudaFree(p);
      if (first == cudaSuccess) first = e;
    }
  delete s;
  if (first != cudaSuccess) return cuda_fail(first, "kdgr_scene_destroy");
  return KDGR_OK;
}

int kdgr_scene_info_get(kdgr_scene_t s, kdgr_scene_info* out) {
  if (!s || !out) {
    set_error("kdgr_scene_info_get: null argument");
    return KDGR_ERR_INVALID_ARG;
  }
  out->n_nodes = s->n_nodes;
  out->n_offsets = s->n_offsets;
  out->n_gaussians = s->n_gauss;
  out->depth = s->depth;
  out->n_leaves = s->n_leaves;
  out->max_leaf = s->max_leaf;
  out->forms = s->forms;
  out->top_nodes = s->top_nodes;
  out->n_aniso = s->n_aniso;
  out->device_bytes = s->device_bytes;
  return KDGR_OK;
}

int kdgr_scene_status(kdgr_scene_t s, uint32_t* bits, int clear) {
  if (!s || !bits) {
    set_error("kdgr_scene_status: null argument");
    return KDGR_ERR_INVALID_ARG;
  }
  DeviceScope on(s->device);
  cudaError_t e = on.err;
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(bits, s->d_status, 4, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && clear) e = cudaMemset(s->d_status, 0, 4);
  if (e != cudaSuccess) return cuda_fail(e, "kdgr_scene_status");
  return KDGR_OK;
}

static int render_common(kdgr_scene_t s, const kdgr_camera* cam, int W, int H, float* rgb, float* alpha, float* depth,
                         kdgr_ray_trace* trace, void* stream, float* ms_out, const char* who) {
  if (!s || !cam || !rgb || W <= 0 || H <= 0) {
    set_error(std::string(who) + ": null scene/camera/output or empty image");
    return KDGR_ERR_INVALID_ARG;
  }
  if (!(s->forms & KDGR_FORM_EXACT)) {
    set_error(std::string(who) + ": scene was created without KDGR_FORM_EXACT");
    return KDGR_ERR_INVALID_ARG;
  }
  DeviceScope on(s->device);
  if (on.err != cudaSuccess) return cuda_fail(on.err, who);
  const cudaStream_t st = (cudaStream_t)stream;
  const CamInfo ci = make_caminfo(*cam, W, H);
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (ms_out) {
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, st);
  }
  cudaError_t e = launch_exact(s->exact_view(), s->plain_view(), ci, W, H, rgb, alpha, depth, trace, s->d_status, st);
  if (e != cudaSuccess) {
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    return cuda_fail(e, who);
  }
  if (ms_out) {
    cudaEventRecord(e1, st);
    e = cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    *ms_out = ms;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (e != cudaSuccess) return cuda_fail(e, who);
  }
  return KDGR_OK;
}

int kdgr_render(kdgr_scene_t s, const kdgr_camera* cam, int W, int H, float* rgb, float* alpha, float* depth,
                void* stream, float* ms_out) {
  return render_common(s, cam, W, H, rgb, alpha, depth, nullptr, stream, ms_out, "kdgr_render");
}

int kdgr_render_trace(kdgr_scene_t s, const kdgr_camera* cam, int W, int H, float* rgb, float* alpha, float* depth,
                      kdgr_ray_trace* trace, void* stream) {
  if (!trace) {
    set_error("kdgr_render_trace: null trace buffer");
    return KDGR_ERR_INVALID_ARG;
  }
  return render_common(s, cam, W, H, rgb, alpha, depth, trace, stream, nullptr, "kdgr_render_trace");
}

}  // extern "C"
