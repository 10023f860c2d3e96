// render_exact.cu -- the plain drop-in render kernel (oracle-matching form).
//
// Replaces renderKernelGaussian_sortNode -> singlePassIntersectGaussian_
// sortNode_onlyShortStack (cudaRenderer.cu:2313-2390, 1488-1709) for the
// hybrid tree (PRIMITIVE_TYPE 2).  Per ray it performs the reference's
// operations in the reference's order, in IEEE round-to-nearest FP32 with no
// fused multiply-add (every operation is an explicit __f*_rn intrinsic), so
// the visited-leaf sequence, the hit sequence and the composited colour match
// the CPU oracle (oracle/oracle.cpp) bit for bit.  The documented deviations
// from the reference binary -- IEEE division instead of __fdividef, 1/sqrt
// instead of rsqrtf, the project exponential instead of CUDA expf -- are the
// oracle's as well.
//
// Two walks give these results:
//   * over the tree as given, one thread per ray (k_render_exact), for traces,
//     for scenes without the leaf-order arrays and for most frames over scenes
//     whose leaf copies outgrow L2: a warp covers an 8x4 pixel tile; the
//     12-entry ring short stack (cudaRenderer.cu:184-210, restart from the root
//     when it runs dry, :1694-1708) lives in shared memory laid out
//     [slot][thread]; Gaussians are an 80-byte test record
//     (reciprocal scale and rotation rows precomputed by the same operations)
//     and a separate 192-byte SH record read only for composited hits;
//   * over the fast form's relaid tree and leaf-order pairs (k_render_plain,
//     render_packet.cuh), as warp packets, independent rays or rays shared by
//     lanes, and by bounced rays (k_render_hybrid): candidates that certainly
//     miss are discarded two at a time in FP32x2 arithmetic with a proven
//     tolerance, the others take the same test as above.  What bounds it is the issue rate, as in the fast form:
//     of 65.1k warp instructions per 8x4 tile (1280x720, 300k Gaussians) the
//     filter on t* leaves 44k and that on the response 34k; 1080p on the 1M
//     scene 4.26 -> 2.39 ms.
// The reference collects every hit of a leaf into a 256-entry local array
// (no overflow check, :1126-1133) and insertion-sorts it.  Here a K-entry
// register buffer keeps the K smallest (t, leaf position) keys; a leaf
// with more than K accepted hits is re-scanned for the next K keys, so any
// leaf size gives the same stable t order with no overflow.
#include <cfloat>
#include <cstdint>

#include "render_packet.cuh"

namespace kdgr {
namespace {

constexpr int kBlock = kThreads;

// Trace-mode counters and sequence hashes of one ray (kdgr_ray_trace).
struct RayStats {
  uint32_t n_inner = 0, n_leaf = 0, n_cand = 0, n_hit = 0, n_blend = 0, n_restart = 0, n_found = 0, max_sort = 0;
  uint64_t hl = kFnvInit, hh = kFnvInit, hb = kFnvInit;
};

// singlePassIntersectGaussian_sortNode_onlyShortStack (cudaRenderer.cu:
// 1488-1709): slab test, descent with the ring stack, per-leaf tests, stable
// hit order, compositing into acc/A/D.  The accumulators are the caller's and
// are not reset, as in the reference (the secondary-ray kernel keeps them
// across bounces).  max_t clips the scene interval (SECONDARY_RAY, :1537-1538;
// FLT_MAX leaves it as is).  Returns false after raising a status bit.
// LEAF: the leaves' candidates are filtered in the leaf-order pairs of L
// (scan_plain), with the same hits accepted, in the same order.
template <int K, bool TRACE, bool LEAF>
__device__ __forceinline__ bool trace_exact(const ExactView& S, const PlainView& L, const F3 o, const F3 d, const float max_t, F3& acc,
                                            float& A, float& D, RayStats& rs, uint32_t (*s_id)[kBlock],
                                            float (*s_t)[kBlock], const int tid, uint32_t* status) {
  float tmin, tmax;
  if (!exact_bounds(S.bmin, S.bmax, o, d, &tmin, &tmax)) return true;
  tmax = fminf(tmax, max_t);
  if (tmin > tmax) return true;
  const float t_scene_far = tmax;
  float t_near = tmin, t_far = tmax;
  uint32_t cur = 0, steps = 0;
  unsigned top = kStack - 1, quant = 0;
  Ray R;  // what scan_plain reads
  R.o = o;
  R.d = d;
  R.oo = dot3(o, o);
  while (A < 0.99f) {
    uint2 nd = __ldg(S.nodes + cur);
    if (++steps > kMaxRaySteps) {
      atomicOr(status, kStatusStepLimit);
      return false;
    }
    while ((nd.x & 7u) != 3u) {
      if (++steps > kMaxRaySteps) {
        atomicOr(status, kStatusStepLimit);
        return false;
      }
      const uint32_t child = nd.x >> 3;
      const uint32_t axis = nd.x & 3u;
      const float o_a = axis == 0 ? o.x : axis == 1 ? o.y : o.z;
      const float d_a = axis == 0 ? d.x : axis == 1 ? d.y : d.z;
      const float t_split = fd(fs(__uint_as_float(nd.y), o_a), d_a);
      const unsigned sign = __float_as_uint(d_a) >> 31;
      const uint32_t idx = child + (sign ^ (t_split <= t_near ? 1u : 0u));
      if (t_near < t_split && t_split < t_far) {
        if (++top == kStack) top = 0;
        quant = min(quant + 1, (unsigned)kStack);
        s_id[top][tid] = child + (sign ^ 1u);
        s_t[top][tid] = t_far;
        t_far = t_split;
      }
      if (child + 1 >= S.n_nodes) {
        atomicOr(status, kStatusBadNode);
        return false;
      }
      if (TRACE) ++rs.n_inner;
      cur = idx;
      nd = __ldg(S.nodes + cur);
    }
    if (TRACE) {
      ++rs.n_leaf;
      rs.hl = fnv_add(rs.hl, cur);
    }
    {
      const uint32_t cnt = nd.x >> 3, base = nd.y;
      if ((uint64_t)base + cnt > S.n_offsets) {
        atomicOr(status, kStatusBadLeaf);
        return false;
      }
      if (TRACE) rs.n_cand += cnt;
      bool have_last = false, saturated = false;
      uint32_t n_acc = 0;  // accepted in this leaf, counted on the first pass
      float last_t = 0.f;
      uint32_t last_i = 0;
      while (true) {
        HitBuf<K> hb;
        hb.clear();
        bool overflow = false;
        if constexpr (LEAF) {
          const LeafRef leaf{__ldg(L.leaf_first + cur), (cnt + 1) >> 1, 0u, 0u};
          R.t_far = t_far;
          uint32_t found = 0;
          overflow = scan_plain<K, 1, false, TRACE>(L, leaf, R, t_near, 0u, have_last, last_t, last_i, hb, &found);
          if (TRACE && !have_last) n_acc = found;
        } else {
          for (uint32_t i = 0; i < cnt; ++i) {
            const uint32_t gid = __ldg(S.offsets + base + i);
            if (gid >= S.n_gauss) {
              atomicOr(status, kStatusBadId);
              return false;
            }
            float t, g;
            if (!exact_test(o, d, S.test + kTestWords * (size_t)gid, t_near, t_far, &t, &g)) continue;
            if (TRACE && !have_last) ++n_acc;
            if (!have_last || t > last_t || (t == last_t && i > last_i)) overflow |= hb.insert(t, g, i);
          }
        }
        // composite the buffered hits in order (cudaRenderer.cu:1611-1687)
#pragma unroll
        for (int k = 0; k < K; ++k) {
          if (hb.t[k] == __int_as_float(0x7f800000)) break;
          const uint32_t gid = __ldg(S.offsets + base + hb.i[k]);
          if (TRACE) {
            ++rs.n_hit;
            rs.hh = fnv_add(rs.hh, gid);
          }
          if (!exact_blend(S.test + kTestWords * (size_t)gid, S.sh + 12ull * gid, d, hb.t[k], hb.g[k], acc, A, D)) continue;
          if (TRACE) {
            ++rs.n_blend;
            rs.hb = fnv_add(rs.hb, gid);
          }
          if (A > 0.99f) {
            saturated = true;
            break;
          }
        }
        if (TRACE && !have_last) {
          rs.n_found += n_acc;
          rs.max_sort = max(rs.max_sort, n_acc);
        }
        if (saturated || !overflow) break;
        have_last = true;
        last_t = hb.t[K - 1];
        last_i = hb.i[K - 1];
      }
    }
    if ((A > 0.99f) | (t_far >= t_scene_far)) break;
    if (quant == 0) {
      cur = 0;
      if (TRACE) ++rs.n_restart;
      t_near = t_far;
      t_far = t_scene_far;
    } else {
      const uint32_t id = s_id[top][tid];
      const float tm = s_t[top][tid];
      if (top == 0) top = kStack;
      --top;
      --quant;
      cur = id;
      t_near = t_far;
      t_far = tm;
    }
  }
  return true;
}

// Blocks from the image middle outwards, unless the walk is packets of 32
// rays: those gain more from neighbouring rows being resident together
// (400k rays, 100k Gaussians: raster order 754 us, middle out 831), the others
// from ending on short rays (256x256: 508, 488).
template <bool RASTER>
__device__ __forceinline__ uint32_t block_order(uint32_t i, uint32_t n) {
  return RASTER ? i : middle_out(i, n);
}

// Pixel of thread `tid` in a 16x8 block: warps cover 8x4 tiles.
template <bool RASTER>
__device__ __forceinline__ void thread_pixel(int tid, int* x, int* y) {
  const int lane = tid & 31, warp = tid >> 5;
  *x = (int)block_order<RASTER>(blockIdx.x, gridDim.x) * 16 + (warp & 1) * 8 + (lane & 7);
  *y = (int)block_order<RASTER>(blockIdx.y, gridDim.y) * 8 + (warp >> 1) * 4 + (lane >> 3);
}

// Ray generation (cudaRenderer.cu:2336-2339): direction through the pixel
// centre, normalised as v * (1 / sqrt(v.v)).
__device__ __forceinline__ F3 primary_dir(const CamInfo& C, int x, int y) {
  const float sx = fa((float)x, 0.5f), sy = fa((float)y, 0.5f);
  const F3 start = mk(C.start[0], C.start[1], C.start[2]);
  const F3 cu = mk(C.u[0], C.u[1], C.u[2]), cv = mk(C.v[0], C.v[1], C.v[2]);
  const F3 o = mk(C.eye[0], C.eye[1], C.eye[2]);
  const F3 dir = sub(add(start, muls(muls(cu, sx), C.step_x)), muls(muls(cv, sy), C.step_y));
  const F3 dv = sub(dir, o);
  return muls(dv, fd(1.f, fq(dot(dv, dv))));
}

__device__ __forceinline__ F3 normalize3(F3 v) { return muls(v, fd(1.f, fq(dot(v, v)))); }

// The plain form (render_packet.cuh): each warp renders one 8x4 tile, or with
// LPR lanes per ray a tile of 32 / LPR rays, of its 16x8 block, as packets
// (PKT) or each lane its own ray.
template <int LPR, int MINB, bool PKT>
__global__ void __launch_bounds__(kThreads, MINB) k_render_plain(PlainView S, CamInfo C, int W, int H, uint32_t n_items,
                                                                 float* __restrict__ rgb,
                                                                 float* __restrict__ alpha_out,
                                                                 float* __restrict__ depth_out, uint32_t* status) {
  __shared__ uint32_t s_id[kStack][kThreads];
  __shared__ float s_t[kStack][kThreads];
  __shared__ PktEnt s_ent[kStack][kWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t it = blockIdx.x * kWarps + warp;
  if (it >= n_items) return;
  const uint32_t blk = it / (4u * LPR), q = it % (4u * LPR), nx = (uint32_t)((W + kBlockW - 1) / kBlockW),
                 ny = (uint32_t)((H + kBlockH - 1) / kBlockH);
  constexpr bool kRaster = PKT && LPR == 1;
  const int bx = (int)block_order<kRaster>(blk % nx, nx) * kBlockW,
            by = (int)block_order<kRaster>(blk / nx, ny) * kBlockH;
  int x, y;
  if constexpr (LPR == 1) block_pixel(KDGR_TILE_8X4, bx, by, (int)q, lane, x, y);
  else group_pixel<LPR>(bx, by, (int)q, lane, x, y);
  const bool inimg = x < W && y < H;
  Ray R;
  R.A = 0.f;
  *acc_slot() = make_float4(0.f, 0.f, 0.f, 0.f);
  const F3 d = primary_dir(C, inimg ? x : 0, inimg ? y : 0);
  const bool live = ray_init_plain(S, mk(C.eye[0], C.eye[1], C.eye[2]), d, FLT_MAX, R) && inimg;
  if constexpr (PKT) {
    trace_packets<kHits, kFormPlain, LPR>(S, R, live, sign_bits(d), s_id, s_t, s_ent, tid, status);
  } else if (live) {
    R.cur = R.steps = 0;
    R.top = kStack - 1;
    R.quant = 0;
    while (R.A < 0.99f && !leaf_step<kHits, kFormPlain, LPR>(S, s_id, s_t, tid, R, status)) {
    }
  }
  if (!inimg || (tid & (LPR - 1)) != 0) return;
  const size_t idx = (size_t)(H - 1 - y) * W + x;  // rows flipped (cudaRenderer.cu:2370)
  const float4 v = *acc_slot();
  rgb[3 * idx] = v.x;
  rgb[3 * idx + 1] = v.y;
  rgb[3 * idx + 2] = v.z;
  if (alpha_out) alpha_out[idx] = R.A;
  if (depth_out) depth_out[idx] = v.w;
}

template <int K, bool TRACE, bool LEAF, int MINB = 0>
__global__ void __launch_bounds__(kBlock, MINB) k_render_exact(ExactView S, PlainView L, CamInfo C, int W, int H, float* __restrict__ rgb,
                                                         float* __restrict__ alpha_out, float* __restrict__ depth_out,
                                                         kdgr_ray_trace* __restrict__ trace, uint32_t* status) {
  __shared__ uint32_t s_id[kStack][kBlock];
  __shared__ float s_t[kStack][kBlock];
  const int tid = threadIdx.x;
  int x, y;
  thread_pixel<false>(tid, &x, &y);
  if (x >= W || y >= H) return;
  const F3 o = mk(C.eye[0], C.eye[1], C.eye[2]);
  const F3 d = primary_dir(C, x, y);
  F3 acc = mk(0.f, 0.f, 0.f);
  float A = 0.f, D = 0.f;
  RayStats rs;
  trace_exact<K, TRACE, LEAF>(S, L, o, d, FLT_MAX, acc, A, D, rs, s_id, s_t, tid, status);
  const size_t idx = (size_t)(H - 1 - y) * W + x;  // rows flipped (cudaRenderer.cu:2370)
  rgb[3 * idx] = acc.x;
  rgb[3 * idx + 1] = acc.y;
  rgb[3 * idx + 2] = acc.z;
  if (alpha_out) alpha_out[idx] = A;
  if (depth_out) depth_out[idx] = D;
  if (TRACE) {
    kdgr_ray_trace tr;
    tr.n_inner = rs.n_inner;
    tr.n_leaf = rs.n_leaf;
    tr.n_cand = rs.n_cand;
    tr.n_hit = rs.n_hit;
    tr.n_blend = rs.n_blend;
    tr.n_restart = rs.n_restart;
    tr.n_found = rs.n_found;
    tr.max_sort = rs.max_sort;
    tr.h_leaf = rs.hl;
    tr.h_hit = rs.hh;
    tr.h_blend = rs.hb;
    trace[(size_t)y * W + x] = tr;
  }
}

// ------------------------------------------------------------ secondary rays
// renderKernelGaussian_Mesh_Hybrid (cudaRenderer.cu:2217-2311): up to five
// bounces; per bounce the closest secondary primitive (spheres,
// intersectSphere :2149-2210, and triangles, intersectTriangleMesh :2114-2147
// with rayTriIntersect :2085-2112) clips the Gaussian pass, then the hit
// reflects, refracts or terminates the ray.  The Gaussian accumulators carry
// over between bounces, as in the reference.
struct SecHit {
  bool hit, front;
  float t;
  F3 n, p;
  int mat;
  float refl, ior;
  F3 color;
};

constexpr float kEps = 0.00001f;  // EPSILON, DefineConst.h:24

__device__ __forceinline__ void sec_material(SecHit& h, const float* m) {
  h.mat = __float_as_int(m[0]);
  h.refl = m[1];
  h.ior = m[2];
  h.color = mk(m[3], m[4], m[5]);
}

__device__ __forceinline__ void sec_set_normal(SecHit& h, const F3 d, F3 n) {
  if (dot(d, n) > 0.0f) {
    h.n = muls(n, -1.0f);
    h.front = false;
  } else {
    h.n = n;
    h.front = true;
  }
}

// Whether a group of triangles may be hit: the line (o, d) passes its sphere
// within a margin.  A triangle test accepts barycentrics in [0, 1] up to its
// rounding, which dividing by |a| >= 1e-5 magnifies: with edges E <= 3.4 and
// s = o - v0 they are off by at most 0.11 E (E + |s|), so a line that the test
// accepts passes the triangle within 3 E times that.
__device__ __forceinline__ bool near_group(const float* __restrict__ g, const F3 o, const F3 d) {
  const float4 c = __ldg(reinterpret_cast<const float4*>(g));
  const float2 e = __ldg(reinterpret_cast<const float2*>(g + 4));  // margin factor, longest edge
  const F3 oc = mk(o.x - c.x, o.y - c.y, o.z - c.z);
  const F3 x = mk(oc.y * d.z - oc.z * d.y, oc.z * d.x - oc.x * d.z, oc.x * d.y - oc.y * d.x);
  const float oc2 = oc.x * oc.x + oc.y * oc.y + oc.z * oc.z;
  const float r = c.w + e.x * (e.y + c.w + sqrtf(oc2));
  return !(x.x * x.x + x.y * x.y + x.z * x.z > 1.001f * r * r + 1e-5f * oc2);
}

// Closest secondary primitive of every active lane's ray; the warp calls it
// together and skips the groups of triangles that none of its rays comes near
// (of 320 triangles of a mirror ball, most tiles of a 720p frame test none:
// 11k of 55k warp instructions per tile before).
__device__ __forceinline__ SecHit intersect_secondary(const HybridView& M, const F3 o, const F3 d, bool active) {
  SecHit h;
  h.hit = false;
  h.t = 1e8f;
  for (int i = 0; i < M.n_spheres; ++i) {
    const float* s = M.spheres + 10 * i;  // center xyz, radius, material words
    const F3 ctr = mk(s[0], s[1], s[2]);
    const F3 oc = sub(o, ctr);
    const float a = dot(d, d);
    const float b = fm(2.0f, dot(oc, d));
    const float c = fs(dot(oc, oc), fm(s[3], s[3]));
    const float disc = fs(fm(b, b), fm(fm(4.0f, a), c));
    if (disc >= 0.0f) {
      const float sq = fq(disc);
      float root = fd(fs(-b, sq), fm(2.0f, a));
      if (root < kEps) root = fd(fa(-b, sq), fm(2.0f, a));
      if (root > kEps && root < h.t) {
        h.hit = true;
        h.t = root;
        h.p = add(o, muls(d, root));
        sec_set_normal(h, d, normalize3(sub(h.p, ctr)));
        sec_material(h, s + 4);
      }
    }
  }
  constexpr uint32_t kSuper = kTriGroup * kTriGroup;
  const uint32_t n_groups = (M.n_tris + kTriGroup - 1) / kTriGroup;
  for (uint32_t first = 0; first < M.n_tris; first += kTriGroup) {
    if (first % kSuper == 0 &&
        !__any_sync(0xFFFFFFFFu, active && near_group(M.groups + 8ull * (n_groups + first / kSuper), o, d))) {
      first += kSuper - kTriGroup;
      continue;
    }
    if (!__any_sync(0xFFFFFFFFu, active && near_group(M.groups + 8ull * (first / kTriGroup), o, d))) continue;
    for (uint32_t i = first; i < min(first + kTriGroup, M.n_tris); ++i) {
      const float* v = M.tris + 9ull * i;
      const F3 v0 = mk(v[0], v[1], v[2]), v1 = mk(v[3], v[4], v[5]), v2 = mk(v[6], v[7], v[8]);
      const F3 e1 = sub(v1, v0), e2 = sub(v2, v0);
      const F3 hv = cross(d, e2);
      const float a = dot(e1, hv);
      if (a > -kEps && a < kEps) continue;
      const float f = fd(1.0f, a);
      const F3 sv = sub(o, v0);
      const float u = fm(f, dot(sv, hv));
      if (u < 0.0f || u > 1.0f) continue;
      const F3 q = cross(sv, e1);
      const float vv = fm(f, dot(d, q));
      if (vv < 0.0f || fa(u, vv) > 1.0f) continue;
      const float t = fm(f, dot(e2, q));
      if (!(t > kEps)) continue;
      if (t < h.t) {
        h.hit = true;
        h.t = t;
        h.p = add(o, muls(d, t));
        sec_set_normal(h, d, normalize3(cross(sub(v1, v0), sub(v2, v0))));
        sec_material(h, M.tri_material);
      }
    }
    __syncwarp();
  }
  return h;
}

// WALK: how the Gaussian passes run -- 0: one thread per ray over the tree as
// given; 1: independent rays over the leaf-order pairs; 2: the primary rays as
// packets, bounced ones independently.  A warp's lanes stay together through
// the bounces; a lane whose ray has ended only waits.  What a pass does not
// need (the running colour, throughput and the hit) waits in shared memory
// meanwhile: in registers it spilled 600 bytes around the walk (WALK 2 with its
// 80 registers still spills 408 / 320 B of stores / loads).
template <int WALK, int MINB>
__global__ void __launch_bounds__(kBlock, MINB)
    k_render_hybrid(ExactView S, PlainView L, CamInfo C, int W, int H, HybridView M, float* __restrict__ rgb,
                    uint32_t* status) {
  __shared__ uint32_t s_id[kStack][kBlock];
  __shared__ float s_t[kStack][kBlock];
  const int tid = threadIdx.x;
  int x, y;
  thread_pixel<WALK == 2>(tid, &x, &y);
  const bool inimg = x < W && y < H;
  F3 o = mk(C.eye[0], C.eye[1], C.eye[2]);
  F3 d = primary_dir(C, inimg ? x : 0, inimg ? y : 0);
  F3 fin = mk(0.f, 0.f, 0.f), thr = mk(1.f, 1.f, 1.f), acc = mk(0.f, 0.f, 0.f);
  constexpr int kKeep = sizeof(SecHit) / 4 + 6;
  static_assert(sizeof(SecHit) % 4 == 0, "SecHit is kept as words");
  __shared__ uint32_t s_keep[WALK == 0 ? 1 : kKeep][kBlock];
  Ray R;  // its opacity, and colour and depth in acc_slot(), carry over between bounces
  R.A = 0.f;
  float D = 0.f;
  if constexpr (WALK != 0) *acc_slot() = make_float4(0.f, 0.f, 0.f, 0.f);
  bool active = inimg;
  for (int bounce = 0; bounce < 5; ++bounce) {
    if (!__any_sync(0xFFFFFFFFu, active)) break;
    SecHit h = intersect_secondary(M, o, d, active);
    const float max_t = h.hit ? h.t : 1e8f;
    if constexpr (WALK == 0) {
      RayStats rs;
      if (active && !trace_exact<8, false, false>(S, L, o, d, max_t, acc, R.A, D, rs, s_id, s_t, tid, status)) active = false;
    } else {
      const bool live = active && ray_init_plain(L, o, d, max_t, R) && R.A < 0.99f;
      uint32_t keep[kKeep];
      memcpy(keep, &h, sizeof h);
      memcpy(keep + sizeof(h) / 4, &fin, 12);
      memcpy(keep + sizeof(h) / 4 + 3, &thr, 12);
#pragma unroll
      for (int k = 0; k < kKeep; ++k) s_keep[k][tid] = keep[k];
      if (WALK == 2 && bounce == 0) {
        __shared__ PktEnt s_ent[kStack][kWarps];
        trace_packets<kHits, kFormPlain, 1>(L, R, live, sign_bits(d), s_id, s_t, s_ent, tid, status);
      } else if (live) {
        R.cur = R.steps = 0;
        R.top = kStack - 1;
        R.quant = 0;
        while (R.A < 0.99f && !leaf_step<kHits, kFormPlain, 1>(L, s_id, s_t, tid, R, status)) {
        }
      }
      __syncwarp();
      const float4 v = *acc_slot();
      acc = mk(v.x, v.y, v.z);
#pragma unroll
      for (int k = 0; k < kKeep; ++k) keep[k] = *(volatile uint32_t*)&s_keep[k][tid];
      memcpy(&h, keep, sizeof h);
      memcpy(&fin, keep + sizeof(h) / 4, 12);
      memcpy(&thr, keep + sizeof(h) / 4 + 3, 12);
      o = R.o;
      d = R.d;
    }
    if (!active) continue;
    const float A = R.A;
    fin = add(fin, mulv(thr, acc));
    thr = muls(thr, fs(1.0f, A));
    if ((thr.x < 0.01f && thr.y < 0.01f && thr.z < 0.01f) || !h.hit) {
      active = false;
      continue;
    }
    const F3 N = h.n, I = d;
    if (h.mat == 1) {  // mirror
      const F3 rdir = sub(I, muls(muls(N, 2.0f), dot(I, N)));
      o = add(h.p, muls(N, 1e-4f));
      d = normalize3(rdir);
      const F3 mc = bounce > 0 ? mk(0.f, 0.f, 0.f) : h.color;
      fin = add(fin, mulv(muls(thr, fs(1.0f, h.refl)), mc));
      thr = muls(thr, h.refl);
    } else if (h.mat == 2) {  // glass
      const float eta = h.front ? fd(1.0f, h.ior) : h.ior;
      const float cos_i = -dot(N, I);
      const float sin_t2 = fm(fm(eta, eta), fs(1.0f, fm(cos_i, cos_i)));
      if (sin_t2 > 1.0f) {  // total internal reflection
        const F3 rdir = sub(I, muls(muls(N, 2.0f), dot(I, N)));
        o = add(h.p, muls(N, 1e-4f));
        d = normalize3(rdir);
      } else {
        const float cos_t = fq(fs(1.0f, sin_t2));
        const F3 tdir = add(muls(I, eta), muls(N, fs(fm(eta, cos_i), cos_t)));
        o = sub(h.p, muls(N, 1e-4f));
        d = normalize3(tdir);
      }
      thr = mulv(thr, h.color);
    } else {  // opaque
      fin = add(fin, mulv(thr, h.color));
      active = false;
    }
  }
  if (!inimg) return;
  const size_t idx = (size_t)(H - 1 - y) * W + x;
  rgb[3 * idx] = fminf(fin.x, 1.0f);
  rgb[3 * idx + 1] = fminf(fin.y, 1.0f);
  rgb[3 * idx + 2] = fminf(fin.z, 1.0f);
}

template <int LPR, int MINB, bool PKT>
cudaError_t launch_plain(const PlainView& s, const CamInfo& cam, int W, int H, float* rgb, float* alpha, float* depth,
                         uint32_t* status, cudaStream_t st) {
  const uint64_t blocks = (uint64_t)((W + kBlockW - 1) / kBlockW) * ((H + kBlockH - 1) / kBlockH);
  if (blocks * LPR > 0x3FFFFFFFull) return cudaErrorInvalidValue;
  k_render_plain<LPR, MINB, PKT><<<(unsigned)(blocks * LPR), kThreads, 0, st>>>(s, cam, W, H, (uint32_t)(blocks * 4 * LPR),
                                                                           rgb, alpha, depth, status);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_exact(const ExactView& s, const PlainView& plain, const CamInfo& cam, int W, int H, float* rgb,
                         float* alpha, float* depth, kdgr_ray_trace* trace, uint32_t* status, cudaStream_t st) {
  if (!trace && plain.leaf_tol) {
    // How the rays are laid on the lanes, by their number (GB300: 152 SMs, 24
    // or 32 resident warps each).  Few rays leave the chip idle and a frame
    // takes as long as its longest ray, so lanes share rays; many rays keep it
    // busy, and the packet walk saves loads and instructions once a tile's
    // rays meet mostly the same leaves.  us over cluster scenes of 10k / 100k
    // / 300k Gaussians, one thread per ray over the tree as given first:
    //   10k rays   257 / 490 / 510   8 lanes, own walk 112 / 196 / 225
    //   40k rays   265 / 486 / 526   4 lanes, packets  176 / 340 / 376   (8 lanes 198 / 437 / 520)
    //   110k rays  246 / 547 / 726   1 lane, own walk  178 / 405 / 475   (packets 233 / 633 / 572)
    //   400k rays  477 / 1215 / 1472 packets           305 / 757 / 880   (own walk 281 / 821 / 1011)
    //   2.1M rays  (1M Gaussians) 4260, packets 2504, with 64 registers 2394
    // The lines over several scenes: at 36k rays 8 lanes and 4-lane packets
    // meet; at 65k packets take 240 (uniform 40k Gaussians) and 413 (cluster
    // 100k), own walks 264 and 366, but uniform scenes would lose against one
    // thread per ray (276); at 307k own walks take 398 / 740, packets 392 / 765.
    // Own walks of one lane have 96 registers: the 80 that 6 blocks leave spill
    // (90k rays, cluster 100k: 409 against 391), 128 leave too few warps (307k:
    // 804 against 740).
    const uint64_t rays = (uint64_t)W * H;
    // Gaussians that sit in more than 64 leaves each: their leaf-order copies
    // outgrow L2 where the records themselves do not (100k overlapping
    // Gaussians, 175 leaves each: 980 MB against 8 MB), so the walk over the
    // tree as given is the faster one unless rays are few (20k rays: 427 us,
    // 8 lanes per ray 198; 250k rays: 540, packets 950, own walk 560) or so many
    // that a packet's rays share most leaves: 2.1M / 3.7M / 8.3M rays over 80k,
    // 100k and 140k overlapping Gaussians (102, 176 and 371 leaves each) 1172 /
    // 1826 / 3598, 1407 / 2190 / 4272 and 1989 / 3058 / 5967 us, packets 1185 /
    // 1588 / 2760, 1471 / 1997 / 3423 and 2322 / 2996 / 4779.
    const bool copies = s.n_offsets / 64u > s.n_gauss;
    if (rays < 36000) return launch_plain<8, 6, false>(plain, cam, W, H, rgb, alpha, depth, status, st);
    if (!copies && rays < 80000) return launch_plain<4, 6, true>(plain, cam, W, H, rgb, alpha, depth, status, st);
    if (!copies && rays < 350000) return launch_plain<1, 5, false>(plain, cam, W, H, rgb, alpha, depth, status, st);
    if (!copies && rays < 1000000) return launch_plain<1, 6, true>(plain, cam, W, H, rgb, alpha, depth, status, st);
    if (!copies || rays >= 3000000) return launch_plain<1, 8, true>(plain, cam, W, H, rgb, alpha, depth, status, st);
  }
  const dim3 grid((W + 15) / 16, (H + 7) / 8);
  // Traces filter the leaves' candidates too, unless the leaf copies are too
  // large for L2 (see above): 640x480, 100k / 10k Gaussians 1310 -> 864 us and
  // 503 -> 309; 256x256 500 -> 373 and 277 -> 199.  A bound of 4 blocks per SM
  // leaves 128 registers (44 B of spills with the filter); without it a 256x256
  // trace takes 397 / 214.
  if (trace && plain.leaf_tol && !(s.n_offsets / 64u > s.n_gauss))
    k_render_exact<8, true, true, 4><<<grid, kBlock, 0, st>>>(s, plain, cam, W, H, rgb, alpha, depth, trace, status);
  else if (trace)
    k_render_exact<8, true, false, 4><<<grid, kBlock, 0, st>>>(s, plain, cam, W, H, rgb, alpha, depth, trace, status);
  // 128 registers pay while every block is resident at once (4 per SM) or
  // nearly: overlapping 100k, 65k / 120k rays 444 / 500 us -> 382 / 432; at
  // 307k rays the blocks wait for each other instead (571 -> 604).
  else if ((uint64_t)W * H < 200000)
    k_render_exact<8, false, false, 4><<<grid, kBlock, 0, st>>>(s, plain, cam, W, H, rgb, alpha, depth, trace, status);
  else
    k_render_exact<8, false, false><<<grid, kBlock, 0, st>>>(s, plain, cam, W, H, rgb, alpha, depth, trace, status);
  return cudaGetLastError();
}

cudaError_t launch_hybrid(const ExactView& s, const PlainView& plain, const CamInfo& cam, int W, int H,
                          const HybridView& m, float* rgb, uint32_t* status, cudaStream_t st) {
  // The walk as in launch_exact; lanes are not shared here (bounced rays part).
  // us with 320 triangles, 100k / 10k Gaussians, one thread per ray first:
  // 256x256 765 / 731, own walk 657 / 599; 1280x720 2352 / 1203, packets
  // 1277 / 967 (own walk 1532 / 933); without groups of triangles to skip the
  // 1280x720 frame took 3400.  Own walks want 128 registers: with 80 they spill
  // and 256x256 with 80 triangles takes 20 % longer, over 20k uniform Gaussians
  // more than the walk over the tree as given (303).  At 500k rays own walks
  // take 523 (uniform 20k) and 1142 (cluster 100k), packets 568 and 1041.
  // Bounced rays gain less from leaf-order pairs than primary ones, so here the
  // tree as given is the faster one from 16 leaves per Gaussian on, for small
  // frames (120k rays over 33k uniform Gaussians, 17 leaves each: 308 us, own
  // walk 339; 26k, 11 leaves each, 81k rays: 256 and 244).
  const dim3 grid((W + 15) / 16, (H + 7) / 8);
  const bool leaf =
      plain.leaf_tol && !(s.n_offsets / ((uint64_t)W * H < 300000 ? 16u : 64u) > s.n_gauss);
  if (!leaf)
    k_render_hybrid<0, 0><<<grid, kBlock, 0, st>>>(s, plain, cam, W, H, m, rgb, status);
  else if ((uint64_t)W * H < 600000)
    k_render_hybrid<1, 4><<<grid, kBlock, 0, st>>>(s, plain, cam, W, H, m, rgb, status);
  else
    k_render_hybrid<2, 6><<<grid, kBlock, 0, st>>>(s, plain, cam, W, H, m, rgb, status);
  return cudaGetLastError();
}

}  // namespace kdgr
