// render_fast.cu -- the batching and precision forms: a persistent kernel
// that draws pixel tiles of many views from an atomic work queue.
//
// Same algorithm as the plain kernel (render_exact.cu): short-stack kd-tree
// traversal front to back, per-leaf max-response test, hits composited in t
// order until the opacity threshold.  What changes, for throughput:
//   * arithmetic: FMA, fast reciprocal, __expf; the ray-Gaussian test reads
//     the precomputed rows of M = diag(1/s) R^T (with b = M mu folded in for
//     the FP32 form), forms ng = M (mu - o) and grdu = M d, accepts t* on
//     the leaf interval without a reciprocal (by the signs of two fused
//     multiply-adds) and only then evaluates the Mahalanobis distance;
//   * hits are accepted with t* in the half-open interval [t_near, t_far),
//     so a Gaussian straddling a split plane is composited in one leaf only;
//   * the tree is relaid out with its top levels breadth-first (they stay
//     hot in L1/L2) and the rest depth-first, and validated at upload, so
//     node steps carry no bounds checks;
//   * the short stack (ring semantics and root restart as the reference) is
//     in shared memory, [slot][thread];
//   * candidate records are stored a second time in leaf order, padded to
//     whole pairs per leaf, so a leaf's candidates are one contiguous run:
//     no ID-then-record dependent load per candidate; the ID is read only
//     for accepted hits;
//   * both forms store leaf entries in interleaved pairs and test them two
//     at a time with Blackwell's packed FP32x2 instructions
//     (fma/mul/add/sub.rn.f32x2), half the arithmetic instructions per test;
//   * warp packets (the default traversal): the 32 rays of a warp tile walk
//     the tree together, each with its own interval and decisions, so a
//     leaf's records are warp-uniform loads (pkt_trace in render_packet.cuh);
//   * lane groups (16, 8 or 4 rays per warp): 2, 4 or 8 lanes hold each ray and
//     split its leaves' candidate pairs, the group taking its hits in key
//     order from the lanes' buffers -- shorter rays and more warps in flight
//     for small batches, the same pixels bit for bit;
//   * pixels are handed out in spatially coherent units (8x4 warp tiles,
//     16x8 CTA blocks, or blocks / tiles from per-SM contiguous strips) so
//     the rays sharing an SM's L1 are neighbours; the autotuner picks the
//     schedule, the register cap (occupancy), the hit-buffer size, the
//     traversal, the warp tile shape and the rays per warp;
//   * precision form: FP16 rows of M with an FP32 mean and BF16 SH (32 + 96
//     bytes per Gaussian instead of 48 + 192); Gaussians whose scale ratio
//     exceeds 1e3 (or whose factors leave the FP16 range) read FP32 factors
//     from the FP64 upload precompute.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <cfloat>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "device_common.cuh"
#include "kdgr_internal.h"
#include "render_packet.cuh"
#include "scene.h"

namespace kdgr {

static_assert(sizeof(ViewDesc) == 96, "ViewDesc layout (bench.py counts 96 B per view)");

namespace {

// Persistent kernel.  Schedules (include/kdgr.h):
//   WARP_TILES: each warp takes `chunk` 8x4 tiles from the global queue;
//   WARP_STRIPS: each warp takes the next quarter of a 16x8 block of
//               its SM's strip of the block list, then steals from the
//               following strips;
//   CTA_BLOCKS: each CTA takes `chunk` 16x8 blocks (barrier per block) and
//               its four warps render the four quarters, so the rays sharing
//               the SM's L1 are neighbours.
// MINB caps registers so that MINB CTAs fit per SM (0: compiler's choice).
// Strip k of n over total items: [total * k / n, total * (k + 1) / n).
__device__ __forceinline__ uint32_t strip_lo(uint32_t total, uint32_t n, uint32_t k) {
  return (uint32_t)((uint64_t)total * k / n);
}

// The first strip after k in visiting order (k + 1, k + 2, ... mod n) whose
// claim counter (queue word 1 + j) is still below its size, or n when every
// strip is exhausted; called by a whole warp.  The lanes read the counters
// together, from L2 (they move by atomics, so not through L1), one load
// each per 32 strips, all issued before the first vote.  Trying the strips
// one claim at a time instead cost a warp up to n sequential atomic round
// trips at the end of a launch, after its last item.  A strip read as open
// may be exhausted by the time the caller claims from it; the caller then
// asks again, and since a counter only grows, every failed claim closes a
// strip for good.
template <typename Open>
__device__ __forceinline__ uint32_t next_open(uint32_t n, uint32_t k, unsigned lane, Open is_open) {
  constexpr int kRounds = (kMaxStrips + 31) / 32;
  bool open[kRounds];
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const uint32_t off = 1u + 32u * r + lane;  // off == n is k itself
    open[r] = off <= n && is_open((k + off) % n);
  }
#pragma unroll
  for (int r = 0; r < kRounds; ++r) {
    const unsigned m = __ballot_sync(0xFFFFFFFFu, open[r]);
    if (m) return (k + 1u + 32u * r + (uint32_t)(__ffs(m) - 1)) % n;
  }
  return n;
}
__device__ __forceinline__ uint32_t next_open_strip(const uint32_t* queue, uint32_t total, uint32_t n, uint32_t k,
                                                    unsigned lane) {
  return next_open(n, k, lane, [&](uint32_t j) {
    return __ldcg(queue + 1 + j) < strip_lo(total, n, j + 1) - strip_lo(total, n, j);
  });
}

// Groups schedule (default configurations; no public value): blocks in groups
// of 2x1 to 2x4, a view's groups numbered by rows and columns from its middle
// outwards and dealt to the SMs in turn, warps claiming quarter blocks of
// their SM's next group and then of the following SMs'.  Against one
// contiguous strip of the block list per SM: every SM gets its share of the
// expensive middle, the packets that start last are the short ones at the
// border, and an SM's resident warps share a squarer piece of the image.  us
// on a GB300, strips first, over cluster scenes: 640x480 of 100k Gaussians 613
// -> 570, 1080p of 1M 1632 -> 1586, 16 mixed views of 300k 10989 -> 10491, packed
// 4x1080p 6884 -> 6777.  One view of 270k to 1M rays over uniform scenes of 3k to
// 20k Gaussians takes 0.87 to 0.93 of the strips' time (geometric means), of 60k
// 1.00, cluster ones 0.92 to 1.01.  Two to nine views gain or lose by how their
// blocks fall on the SMs, single launches between 0.74 and 1.32, on average 0.98
// (cluster) and 1.02 (uniform); eleven other deals (group sizes, raster order,
// contiguous runs) spread as much.  Smaller groups balance small launches
// better, larger ones share more of the L1 (640x480: 2x1 541, 2x2 574, 2x4 592;
// mixed: 10582, 10453, 10393).
struct GroupShape {
  uint32_t lx, ly;  // blocks of a group, as powers of two
};
GroupShape group_shape(uint64_t tiles) {  // by the launch's 8x4 tiles
  return tiles < 16384u ? GroupShape{1, 0} : tiles < 131072u ? GroupShape{1, 1} : GroupShape{1, 2};
}
// `chunk` argument of a groups launch: SMs, lx, ly.
int group_arg(int sms, GroupShape g) { return sms | (int)(g.lx << 16 | g.ly << 20); }

// A warp's place in the dealt groups.
struct GroupWalk {
  uint32_t n, lx, ly, groups, per;  // SMs, group shape, groups of the launch, items of a group
  uint32_t k, fails;                // whose groups the warp claims from; exhausted ones it has met
  __device__ __forceinline__ GroupWalk(int arg, uint32_t total, uint32_t items_per_block)
      : n((uint32_t)arg & 0xFFFFu), lx(((uint32_t)arg >> 16) & 15u), ly((uint32_t)arg >> 20), groups(total),
        per(items_per_block << (lx + ly)), fails(0) {
    uint32_t smid;
    asm("mov.u32 %0, %%smid;" : "=r"(smid));
    k = smid % n;
  }
  __device__ __forceinline__ uint32_t items(uint32_t j) const { return j < groups ? (groups - j + n - 1) / n * per : 0u; }
  // The warp's next item: its group and its number inside; false when every
  // group is taken.  queue word 1 + j counts the claims from SM j's groups; an
  // exhausted SM is followed by the first with items left, as next_open_strip.
  __device__ __forceinline__ bool next(uint32_t* queue, unsigned lane, uint32_t& group, uint32_t& sub) {
    while (fails <= n) {
      uint32_t c = 0;
      if (lane == 0) c = atomicAdd(queue + 1 + k, 1u);
      c = __shfl_sync(0xFFFFFFFFu, c, 0);
      if (c < items(k)) {
        group = c / per * n + k;
        sub = c % per;
        return true;
      }
      ++fails;
      k = next_open(n, k, lane, [&](uint32_t j) { return __ldcg(queue + 1 + j) < items(j); });
      if (k >= n) return false;
    }
    return false;
  }
  // Top-left pixel of block `b` of group `lg` of a W x H view.
  __device__ __forceinline__ void block(uint32_t lg, uint32_t b, int W, int H, int& bx, int& by) const {
    const uint32_t gx = ((uint32_t)W + (16u << lx) - 1) >> (4 + lx), gy = ((uint32_t)H + (8u << ly) - 1) >> (3 + ly);
    bx = (int)(middle_out(lg % gx, gx) << (4 + lx)) + (int)(b & ((1u << lx) - 1u)) * kBlockW;
    by = (int)(middle_out(lg / gx, gy) << (3 + ly)) + (int)(b >> lx) * kBlockH;
  }
};

template <bool PACKED, int SCHED, int MINB, int KB, bool PKT, int LPR>
__global__ void __launch_bounds__(kThreads, MINB) k_render_batch(FastView S, const ViewDesc* __restrict__ views,
                                                                 int n_views, uint32_t total_items,
                                                                 float* __restrict__ rgb,
                                                                 float* __restrict__ alpha_out,
                                                                 float* __restrict__ depth_out, uint32_t* queue,
                                                                 uint32_t* status, int chunk, int tile) {
  __shared__ uint32_t s_id[kStack][kThreads];
  __shared__ float s_t[kStack][kThreads];
  __shared__ PktEnt s_ent[kStack][kWarps];
  __shared__ uint32_t s_work;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if constexpr (SCHED == kSchedGroups) {
    GroupWalk G(chunk, total_items, 4u * LPR);
    uint32_t g, sub;
    while (G.next(queue, (unsigned)lane, g, sub)) {
      const ViewDesc& V = views[find_view(views, n_views, g, kSchedGroups)];
      const int W = __ldg(&V.W), H = __ldg(&V.H);
      int bx, by, x, y;
      G.block(g - __ldg(&V.grp_base), sub / (4u * LPR), W, H, bx, by);
      if (bx >= W || by >= H) continue;  // a group's blocks beyond the image
      const int q = (int)(sub % (4u * LPR));
      if constexpr (LPR == 1) block_pixel(tile, bx, by, q, lane, x, y);
      else group_pixel<LPR>(bx, by, q, lane, x, y);
      render_px<KB, PACKED ? kFormPacked : kFormFp32, PKT, LPR>(S, V, x, y, s_id, s_t, s_ent, tid, rgb, alpha_out,
                                                                depth_out, status);
    }
  } else if constexpr (SCHED == KDGR_SCHED_WARP_STRIPS) {
    // items are quarters of 16x8 blocks (warp tiles in block order), or with
    // LPR lanes per ray 4 LPR tiles of 32 / LPR rays; each warp claims the
    // next item of its SM's strip, no CTA barrier
    uint32_t smid;
    asm("mov.u32 %0, %%smid;" : "=r"(smid));
    const uint32_t n = (uint32_t)chunk;  // number of strips
    uint32_t k = smid % n, fails = 0;
    while (fails <= n) {  // a warp's claims fail at most once per strip
      const uint32_t b0 = strip_lo(total_items, n, k), b1 = strip_lo(total_items, n, k + 1);
      uint32_t it = 0;
      if (lane == 0) it = b0 + atomicAdd(queue + 1 + k, 1u);
      it = __shfl_sync(0xFFFFFFFFu, it, 0);
      if (it >= b1) {
        ++fails;
        k = next_open_strip(queue, total_items, n, k, (unsigned)lane);
        if (k >= n) break;
        continue;
      }
      const uint32_t blk = it / (4u * LPR), q = it % (4u * LPR);
      const ViewDesc& V = views[find_view(views, n_views, blk, KDGR_SCHED_CTA_BLOCKS)];
      const uint32_t lb = blk - __ldg(&V.cb_base), nx = __ldg(&V.cb_x);
      int x, y;
      if constexpr (LPR == 1) block_pixel(tile, (int)(lb % nx) * kBlockW, (int)(lb / nx) * kBlockH, (int)q, lane, x, y);
      else group_pixel<LPR>((int)(lb % nx) * kBlockW, (int)(lb / nx) * kBlockH, (int)q, lane, x, y);
      render_px<KB, PACKED ? kFormPacked : kFormFp32, PKT, LPR>(S, V, x, y, s_id, s_t, s_ent, tid, rgb, alpha_out, depth_out,
                                      status);
    }
  } else if constexpr (SCHED == KDGR_SCHED_SM_STRIPS) {
    // strip of this SM: [total * k / n, total * (k + 1) / n), k = smid mod n
    __shared__ uint32_t s_strip;
    uint32_t smid;
    asm("mov.u32 %0, %%smid;" : "=r"(smid));
    const uint32_t n = (uint32_t)chunk;  // number of strips (the SM count; chunk is reused for it)
    if (tid == 0) s_strip = smid % n;
    while (true) {
      __syncthreads();
      if (warp == 0) {
        // claim the next item of this CTA's strip, or move on to the next
        // strip with items left (a failed claim closes its strip for good)
        uint32_t k = s_strip, item = 0xFFFFFFFFu;
        for (uint32_t fails = 0; fails <= n; ++fails) {
          const uint32_t b0 = strip_lo(total_items, n, k), b1 = strip_lo(total_items, n, k + 1);
          uint32_t it = 0;
          if (lane == 0) it = b0 + atomicAdd(queue + 1 + k, 1u);
          it = __shfl_sync(0xFFFFFFFFu, it, 0);
          if (it < b1) {
            item = it;
            break;
          }
          k = next_open_strip(queue, total_items, n, k, (unsigned)lane);
          if (k >= n) break;
        }
        if (lane == 0) {
          s_work = item;
          if (k < n) s_strip = k;
        }
      }
      __syncthreads();
      const uint32_t item = s_work;
      if (item == 0xFFFFFFFFu) break;
      const ViewDesc& V = views[find_view(views, n_views, item, KDGR_SCHED_CTA_BLOCKS)];
      const uint32_t lb = item - __ldg(&V.cb_base), nx = __ldg(&V.cb_x);
      int x, y;
      block_pixel(tile, (int)(lb % nx) * kBlockW, (int)(lb / nx) * kBlockH, warp, lane, x, y);
      render_px<KB, PACKED ? kFormPacked : kFormFp32, PKT, 1>(S, V, x, y, s_id, s_t, s_ent, tid, rgb, alpha_out, depth_out, status);
    }
  } else {
    while (true) {
      uint32_t first;
      if constexpr (SCHED == KDGR_SCHED_CTA_BLOCKS) {
        __syncthreads();
        if (tid == 0) s_work = atomicAdd(queue, (uint32_t)chunk);
        __syncthreads();
        first = s_work;
      } else {
        uint32_t f = 0;
        if (lane == 0) f = atomicAdd(queue, (uint32_t)chunk);
        first = __shfl_sync(0xFFFFFFFFu, f, 0);
      }
      if (first >= total_items) break;
      const uint32_t last = min(first + (uint32_t)chunk, total_items);
      for (uint32_t item = first; item < last; ++item) {
        const ViewDesc& V = views[find_view(views, n_views, item, SCHED)];
        int x, y;
        if (SCHED == KDGR_SCHED_CTA_BLOCKS) {
          const uint32_t lb = item - __ldg(&V.cb_base), nx = __ldg(&V.cb_x);
          block_pixel(tile, (int)(lb % nx) * kBlockW, (int)(lb / nx) * kBlockH, warp, lane, x, y);
        } else {
          const uint32_t lt = item - __ldg(&V.wt_base), nx = __ldg(&V.wt_x);
          x = (int)(lt % nx) * kTileW + (lane & 7);
          y = (int)(lt / nx) * kTileH + (lane >> 3);
        }
        render_px<KB, PACKED ? kFormPacked : kFormFp32, PKT, 1>(S, V, x, y, s_id, s_t, s_ent, tid, rgb, alpha_out, depth_out, status);
      }
    }
  }
}

// Multi-scene form for the serving loop: every view names a scene slot and
// each warp renders its quarter-block against that slot's arrays (the slot
// table travels in the launch parameters, so the warp-uniform field reads hit
// the constant cache).  One persistent launch serves the requests of all
// resident scenes queued in a tick.  outs[v] is view v's output base (the
// device arena, or a request's page-locked host buffer); the view's out_off
// counts pixels from it.  PKT, LPR: the walk, as in k_render_batch; items are
// dealt by groups, or with lanes sharing rays taken from warp strips (`share`
// and `total` as the schedules' chunk and total_items).
template <bool PACKED, int MINB, bool PKT, int LPR>
__global__ void __launch_bounds__(kThreads, MINB) k_render_multi(const __grid_constant__ SceneTable scenes,
                                                              const ViewDesc* __restrict__ views, int n_views,
                                                              uint32_t total, float* const* __restrict__ outs,
                                                              uint32_t* queue, uint32_t* status, int share) {
  __shared__ uint32_t s_id[kStack][kThreads];
  __shared__ float s_t[kStack][kThreads];
  __shared__ PktEnt s_ent[kStack][kWarps];
  const int tid = threadIdx.x, lane = tid & 31;
  auto render = [&](int vi, int bx, int by, int q) {
    const ViewDesc& V = views[vi];
    const FastView& S = scenes.s[__ldg(&V.scene) & (kSceneSlots - 1)];
    int x, y;
    if constexpr (LPR == 1) block_pixel(KDGR_TILE_8X4, bx, by, q, lane, x, y);
    else group_pixel<LPR>(bx, by, q, lane, x, y);
    render_px<kHits, PACKED ? kFormPacked : kFormFp32, PKT, LPR>(S, V, x, y, s_id, s_t, s_ent, tid, outs[vi], nullptr,
                                                                nullptr, status);
  };
  if constexpr (LPR == 1) {
    GroupWalk G(share, total, 4u);
    uint32_t g, sub;
    while (G.next(queue, (unsigned)lane, g, sub)) {
      const int vi = find_view(views, n_views, g, kSchedGroups);
      const int W = __ldg(&views[vi].W), H = __ldg(&views[vi].H);
      int bx, by;
      G.block(g - __ldg(&views[vi].grp_base), sub / 4u, W, H, bx, by);
      if (bx < W && by < H) render(vi, bx, by, (int)(sub % 4u));
    }
  } else {
    uint32_t smid;
    asm("mov.u32 %0, %%smid;" : "=r"(smid));
    const uint32_t n = (uint32_t)share;
    uint32_t k = smid % n, fails = 0;
    while (fails <= n) {  // a warp's claims fail at most once per strip
      const uint32_t b0 = strip_lo(total, n, k), b1 = strip_lo(total, n, k + 1);
      uint32_t it = 0;
      if (lane == 0) it = b0 + atomicAdd(queue + 1 + k, 1u);
      it = __shfl_sync(0xFFFFFFFFu, it, 0);
      if (it >= b1) {
        ++fails;
        k = next_open_strip(queue, total, n, k, (unsigned)lane);
        if (k >= n) break;
        continue;
      }
      const uint32_t blk = it / (4u * LPR);
      const int vi = find_view(views, n_views, blk, KDGR_SCHED_CTA_BLOCKS);
      const uint32_t lb = blk - __ldg(&views[vi].cb_base), nx = __ldg(&views[vi].cb_x);
      render(vi, (int)(lb % nx) * kBlockW, (int)(lb / nx) * kBlockH, (int)(it % (4u * LPR)));
    }
  }
}

// FP64 precompute of M = diag(1/s) R^T and b = M mu for anisotropic
// Gaussians (upload time only).  src: 10 floats per entry (inverse scale x3,
// quaternion w,x,y,z, mean x3).
__global__ void k_aniso_fp64(const float* __restrict__ src, uint32_t n, float4* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* p = src + 10ull * i;
  double r = p[3], x = p[4], y = p[5], z = p[6];
  const double qn = 1.0 / sqrt(r * r + x * x + y * y + z * z);
  r *= qn;
  x *= qn;
  y *= qn;
  z *= qn;
  const double xx = x * x, yy = y * y, zz = z * z, xy = x * y, xz = x * z, yz = y * z;
  const double rx = r * x, ry = r * y, rz = r * z;
  const double m[3][3] = {{1 - 2 * (yy + zz), 2 * (xy + rz), 2 * (xz - ry)},
                          {2 * (xy - rz), 1 - 2 * (xx + zz), 2 * (yz + rx)},
                          {2 * (xz + ry), 2 * (yz - rx), 1 - 2 * (xx + yy)}};
  for (int row = 0; row < 3; ++row) {
    const double s = p[row];
    const double a = s * m[row][0], b = s * m[row][1], c = s * m[row][2];
    const double bb = a * p[7] + b * p[8] + c * p[9];
    out[3ull * i + row] = make_float4((float)a, (float)b, (float)c, (float)bb);
  }
}

using KernelFn = void (*)(FastView, const ViewDesc*, int, uint32_t, float*, float*, float*, uint32_t*, uint32_t*,
                          int, int);

template <bool PACKED, int SCHED, int KB, bool PKT, int LPR>
KernelFn pick_minb(int minb) {
  if (minb >= 8) return k_render_batch<PACKED, SCHED, 8, KB, PKT, LPR>;
  if (minb >= 6) return k_render_batch<PACKED, SCHED, 6, KB, PKT, LPR>;
  return k_render_batch<PACKED, SCHED, 0, KB, PKT, LPR>;
}

// Lanes per ray: 32 / rays_per_warp (warp-strip schedule only; 4 rays per
// warp only from choose_walk).
int lanes_per_ray(const kdgr_batch_config& c) {
  return c.rays_per_warp == 4 ? 8 : c.rays_per_warp == 8 ? 4 : c.rays_per_warp == 16 ? 2 : 1;
}

template <bool PACKED, int KB, bool PKT>
KernelFn pick_sched_k(const kdgr_batch_config& c) {
  if constexpr (KB == kHits)  // choose_walk's launches only: packets with 64 registers, independent rays with 80
    if (c.schedule == kSchedGroups) return k_render_batch<PACKED, kSchedGroups, PKT ? 8 : 6, KB, PKT, 1>;
  if (c.schedule == KDGR_SCHED_CTA_BLOCKS) return pick_minb<PACKED, KDGR_SCHED_CTA_BLOCKS, KB, PKT, 1>(c.min_blocks);
  if (c.schedule == KDGR_SCHED_SM_STRIPS) return pick_minb<PACKED, KDGR_SCHED_SM_STRIPS, KB, PKT, 1>(c.min_blocks);
  if (c.schedule == KDGR_SCHED_WARP_STRIPS) {
    if constexpr (KB == kHits && PKT)  // choose_walk's small launches only
      if (lanes_per_ray(c) == 8) return k_render_batch<PACKED, KDGR_SCHED_WARP_STRIPS, 6, KB, PKT, 8>;
    if (lanes_per_ray(c) == 4) return pick_minb<PACKED, KDGR_SCHED_WARP_STRIPS, KB, PKT, 4>(c.min_blocks);
    if (lanes_per_ray(c) == 2) return pick_minb<PACKED, KDGR_SCHED_WARP_STRIPS, KB, PKT, 2>(c.min_blocks);
    return pick_minb<PACKED, KDGR_SCHED_WARP_STRIPS, KB, PKT, 1>(c.min_blocks);
  }
  return pick_minb<PACKED, KDGR_SCHED_WARP_TILES, KB, PKT, 1>(c.min_blocks);
}

template <bool PACKED, bool PKT>
KernelFn pick_sched_t(const kdgr_batch_config& c) {
  return c.hit_buffer == 8 ? pick_sched_k<PACKED, 8, PKT>(c) : pick_sched_k<PACKED, kHits, PKT>(c);
}

template <bool PACKED>
KernelFn pick_sched(const kdgr_batch_config& c) {
  return c.traversal == KDGR_TRAV_RAY ? pick_sched_t<PACKED, false>(c) : pick_sched_t<PACKED, true>(c);
}

KernelFn pick_kernel(const kdgr_batch_config& c) {
  return c.precision ? pick_sched<true>(c) : pick_sched<false>(c);
}

// SM count of the current device, cached per device.  Threads may race on
// the first query of a device; they all store the same value.
constexpr int kMaxSmCacheDevices = 64;
std::atomic<int> g_num_sms[kMaxSmCacheDevices];

int num_sms() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = -1;
  const bool cacheable = dev >= 0 && dev < kMaxSmCacheDevices;
  if (cacheable) n = g_num_sms[dev].load(std::memory_order_relaxed);
  if (n > 0) return n;
  if (dev < 0 || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 1;
  if (cacheable) g_num_sms[dev].store(n, std::memory_order_relaxed);
  return n;
}

// Resident 128-thread CTAs per SM of a kernel on the current device (at
// least 1), cached per kernel and device: the query costs microseconds and
// every batched launch needs it.
cudaError_t resident_ctas(const void* fn, int* out) {
  static std::mutex mu;
  static std::vector<std::pair<std::pair<const void*, int>, int>> cache;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  {
    std::lock_guard<std::mutex> lk(mu);
    for (const auto& it : cache)
      if (it.first.first == fn && it.first.second == dev) {
        *out = it.second;
        return cudaSuccess;
      }
  }
  int occ = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kThreads, 0);
  if (e != cudaSuccess) return e;
  occ = occ > 0 ? occ : 1;
  std::lock_guard<std::mutex> lk(mu);
  cache.push_back({{fn, dev}, occ});
  *out = occ;
  return cudaSuccess;
}
template <typename F>
cudaError_t resident_ctas(F* fn, int* out) {
  return resident_ctas(reinterpret_cast<const void*>(fn), out);
}

}  // namespace

// First group of every view and their number, for a launch of `tiles` 8x4
// tiles in all.
uint32_t number_groups(ViewDesc* views, int n_views, uint64_t tiles) {
  const GroupShape gs = group_shape(tiles);
  uint64_t base = 0;
  for (int v = 0; v < n_views; ++v) {
    views[v].grp_base = (uint32_t)base;
    base += (uint64_t)((views[v].W + (16 << gs.lx) - 1) >> (4 + gs.lx)) *
            (uint64_t)((views[v].H + (8 << gs.ly) - 1) >> (3 + gs.ly));
  }
  return (uint32_t)base;
}

// Host: view table and total tile count for a list of views.
int make_view_table(const kdgr_view* views, int n_views, std::vector<ViewDesc>& out, uint32_t totals[3]) {
  out.resize(n_views);
  return fill_view_table(views, n_views, out.data(), totals);
}

// The view table of n_views views into a caller-provided array (no
// allocation); make_view_table and the allocation-free entry point share it.
int fill_view_table(const kdgr_view* views, int n_views, ViewDesc* out, uint32_t totals[3]) {
  uint64_t wbase = 0, cbase = 0;
  for (int v = 0; v < n_views; ++v) {
    const kdgr_view& kv = views[v];
    if (kv.width <= 0 || kv.height <= 0) {
      set_error("view " + std::to_string(v) + " has an empty image");
      return KDGR_ERR_INVALID_ARG;
    }
    ViewDesc& d = out[v];
    d.cam = make_caminfo(kv.cam, kv.width, kv.height);
    d.W = kv.width;
    d.H = kv.height;
    d.wt_x = (uint32_t)((kv.width + kTileW - 1) / kTileW);
    d.wt_base = (uint32_t)wbase;
    d.cb_x = (uint32_t)((kv.width + kBlockW - 1) / kBlockW);
    d.cb_base = (uint32_t)cbase;
    d.out_off = kv.out_offset;
    d.scene = 0;
    d.grp_base = 0;
    wbase += (uint64_t)d.wt_x * (uint64_t)((kv.height + kTileH - 1) / kTileH);
    cbase += (uint64_t)d.cb_x * (uint64_t)((kv.height + kBlockH - 1) / kBlockH);
    if (wbase > 0xF0000000ull) {
      set_error("batch too large: more than 2^32 tiles");
      return KDGR_ERR_LIMIT;
    }
  }
  totals[0] = (uint32_t)wbase;
  totals[1] = (uint32_t)cbase;
  totals[2] = number_groups(out, n_views, wbase);
  return KDGR_OK;
}

int check_batch_config(kdgr_scene_t s, const kdgr_batch_config& c) {
  if (c.precision && !(s->forms & KDGR_FORM_PACKED)) {
    set_error("precision form requested but the scene was created without KDGR_FORM_PACKED");
    return KDGR_ERR_INVALID_ARG;
  }
  if (!c.precision && !(s->forms & KDGR_FORM_FAST)) {
    set_error("FP32 fast form requested but the scene was created without KDGR_FORM_FAST");
    return KDGR_ERR_INVALID_ARG;
  }
  if (c.chunk < 1 || c.chunk > 64) {
    set_error("batch config: chunk must be in 1..64");
    return KDGR_ERR_INVALID_ARG;
  }
  if (c.schedule != KDGR_SCHED_WARP_TILES && c.schedule != KDGR_SCHED_CTA_BLOCKS &&
      c.schedule != KDGR_SCHED_SM_STRIPS && c.schedule != KDGR_SCHED_WARP_STRIPS) {
    set_error("batch config: unknown schedule");
    return KDGR_ERR_INVALID_ARG;
  }
  if (c.hit_buffer != 0 && c.hit_buffer != 4 && c.hit_buffer != 8) {
    set_error("batch config: hit_buffer must be 0, 4 or 8");
    return KDGR_ERR_INVALID_ARG;
  }
  if (c.min_blocks != 0 && c.min_blocks != 6 && c.min_blocks != 8) {
    set_error("batch config: min_blocks must be 0, 6 or 8");
    return KDGR_ERR_INVALID_ARG;
  }
  if (c.tile_shape != KDGR_TILE_8X4 && c.tile_shape != KDGR_TILE_4X8 && c.tile_shape != KDGR_TILE_16X2) {
    set_error("batch config: tile_shape must be KDGR_TILE_8X4, KDGR_TILE_4X8 or KDGR_TILE_16X2");
    return KDGR_ERR_INVALID_ARG;
  }
  if (c.tile_shape != KDGR_TILE_8X4 && c.schedule == KDGR_SCHED_WARP_TILES) {
    set_error("batch config: the warp-tile schedule renders 8x4 tiles only");
    return KDGR_ERR_INVALID_ARG;
  }
  if (c.traversal != KDGR_TRAV_PACKET && c.traversal != KDGR_TRAV_RAY) {
    set_error("batch config: traversal must be KDGR_TRAV_PACKET or KDGR_TRAV_RAY");
    return KDGR_ERR_INVALID_ARG;
  }
  if (c.rays_per_warp != 0 && c.rays_per_warp != 32 && c.rays_per_warp != 16 && c.rays_per_warp != 8) {
    set_error("batch config: rays_per_warp must be 0, 32, 16 or 8");
    return KDGR_ERR_INVALID_ARG;
  }
  if (lanes_per_ray(c) > 1 && (c.schedule != KDGR_SCHED_WARP_STRIPS || c.tile_shape != KDGR_TILE_8X4)) {
    set_error("batch config: 16 or 8 rays per warp need the warp-strip schedule and the default tile shape");
    return KDGR_ERR_INVALID_ARG;
  }
  return KDGR_OK;
}

// How few rays a launch may have before its walk changes.  One frame of R rays
// on the default walk (packets of 32 rays, 64 registers) takes as long as its
// longest packet when R is small; us on a GB300, default first, over cluster
// scenes of 10k / 100k / 300k Gaussians and a dense uniform one (100k):
//   10k rays   349 / 891 / 799 / 1670   4-ray packets 115 / 206 / 200 / 270
//   40k rays   246 / 596 / 535 / 1438   own walk      160 / 298 / 334 / 293   (4-ray packets 177 / 325 / 356 / 312)
//   160k rays  234 / 526 / 458 / 1099   own walk      194 / 424 / 446 / 401
//   400k rays  282 / 629 / 696 / 783    own walk      282 / 650 / 748 / 521
// A scene whose Gaussians sit in more than 64 leaves each (the last one) has
// leaves far smaller than a tile: its rays share too few of them for packets
// up to a full frame (1.1M rays: 924 us, own walk 850).  Between 16 and 64
// leaves each, own walks win less far up; uniform 33k / 40k / 55k Gaussians (17,
// 22 and 40 leaves each), packets and own walk: one frame of 307k rays 264 / 284
// / 329 and 237 / 247 / 276; 6 views of 88k rays, packed, 627 / 713 / 981 and
// 443 / 454 / 494; one frame of 858k rays 350 / 381 / 441 and 390 / 398 / 439.
// At 11 leaves each one frame is as fast either way (233, 217).
constexpr uint64_t kFewRays = 30000, kSomeRays = 250000, kSomeRaysMid = 600000, kSomeRaysDense = 1200000;

// The configuration a launch runs with: a caller's own choice as it is; the
// default one (precision apart) by groups, with the walk that suits the number
// of rays.
// Every walk gives the same pixels bit for bit.
kdgr_batch_config choose_walk(kdgr_scene_t s, const kdgr_batch_config& c, uint64_t rays) {
  kdgr_batch_config d;
  kdgr_batch_config_default(&d);
  d.precision = c.precision;
  kdgr_batch_config n = c;  // with the values that 0 stands for
  if (n.hit_buffer == 0) n.hit_buffer = 4;
  if (n.rays_per_warp == 0) n.rays_per_warp = 32;
  if (memcmp(&d, &n, sizeof d) != 0) return c;
  const bool mid = s->n_pair_entries / 16u > s->n_gauss, dense = s->n_pair_entries / 64u > s->n_gauss;
  d.schedule = kSchedGroups;
  if (rays >= (dense ? kSomeRaysDense : mid ? kSomeRaysMid : kSomeRays)) return d;
  d.min_blocks = 6;
  if (rays < kFewRays) {
    d.schedule = KDGR_SCHED_WARP_STRIPS;  // the finest shares: 10k rays 210 us, in groups 275
    d.rays_per_warp = 4;
  } else {
    d.traversal = KDGR_TRAV_RAY;
  }
  return d;
}

// Launch the persistent kernel.  `queue` must read 0 when the kernel starts.
cudaError_t launch_batch(kdgr_scene_t s, const kdgr_batch_config& cc, const ViewDesc* d_views, int n_views,
                         const uint32_t totals[3], float* rgb, float* alpha, float* depth, uint32_t* queue,
                         cudaStream_t st) {
  const kdgr_batch_config c = choose_walk(s, cc, 32ull * totals[0]);
  const bool by_groups = c.schedule == kSchedGroups;
  const uint32_t total_tiles = totals[0], total_blocks = totals[1];
  KernelFn fn = pick_kernel(c);
  int per_sm = c.blocks_per_sm;
  if (per_sm <= 0) {
    cudaError_t e = resident_ctas(fn, &per_sm);
    if (e != cudaSuccess) return e;
  }
  const bool warp_strips = c.schedule == KDGR_SCHED_WARP_STRIPS;
  const bool per_warp = c.schedule == KDGR_SCHED_WARP_TILES || warp_strips;
  if (warp_strips && total_blocks > 0x3FFFFFFFu) return cudaErrorInvalidValue;
  const uint32_t lpr = (uint32_t)lanes_per_ray(c);
  if (warp_strips && total_blocks > 0x3FFFFFFFu / lpr) return cudaErrorInvalidValue;
  const uint32_t total =
      by_groups ? totals[2] : warp_strips ? 4u * lpr * total_blocks : per_warp ? total_tiles : total_blocks;
  // SM strips: the kernel's `chunk` argument carries the number of strips
  const bool strips = c.schedule == KDGR_SCHED_SM_STRIPS || warp_strips || by_groups;
  const GroupShape gs = group_shape(total_tiles);
  int chunk = strips ? std::min(num_sms(), kMaxStrips) : c.chunk;
  if (by_groups) chunk = group_arg(chunk, gs);
  uint64_t blocks = (uint64_t)num_sms() * per_sm;
  const uint64_t grabs = strips ? total : ((uint64_t)total + chunk - 1) / chunk;
  const uint64_t cap = by_groups ? ((uint64_t)lpr << (gs.lx + gs.ly)) * total : per_warp ? (grabs + kWarps - 1) / kWarps : grabs;
  if (blocks > cap) blocks = cap > 0 ? cap : 1;
  fn<<<(unsigned)blocks, kThreads, 0, st>>>(s->fast_view(c.precision != 0), d_views, n_views, total, rgb, alpha,
                                            depth, queue, s->d_status, chunk, c.tile_shape);
  return cudaGetLastError();
}

// Pair p of the packed plain records (layout at PPairRec) from the
// per-Gaussian staging words: mean x, y, z (FP32), half2 (M22, 0),
// half2 (M00, M01), (M02, M10), (M11, M12), (M20, M21).  Padding entries
// are zero.
__global__ void k_build_ppairs(const uint32_t* __restrict__ gid, uint32_t n, const uint32_t* __restrict__ src,
                               uint4* __restrict__ out) {
  const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= (size_t)n / 2) return;
  uint32_t a[8], b[8];
  const uint32_t g0 = __ldg(gid + 2 * p), g1 = __ldg(gid + 2 * p + 1);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    a[i] = g0 == kPadGid ? 0u : __ldg(src + 8ull * g0 + i);
    b[i] = g1 == kPadGid ? 0u : __ldg(src + 8ull * g1 + i);
  }
  auto lo = [](uint32_t x) { return x & 0xFFFFu; };
  auto hi = [](uint32_t x) { return x >> 16; };
  auto h2 = [](uint32_t l, uint32_t h) { return l | (h << 16); };
  out[4 * p] = make_uint4(a[0], b[0], a[1], b[1]);
  out[4 * p + 1] = make_uint4(a[2], b[2], h2(lo(a[4]), lo(b[4])), h2(hi(a[4]), hi(b[4])));
  out[4 * p + 2] = make_uint4(h2(lo(a[5]), lo(b[5])), h2(hi(a[5]), hi(b[5])), h2(lo(a[6]), lo(b[6])),
                              h2(hi(a[6]), hi(b[6])));
  out[4 * p + 3] = make_uint4(h2(lo(a[7]), lo(b[7])), h2(hi(a[7]), hi(b[7])), h2(lo(a[3]), lo(b[3])), 0u);
}

// Pair p of the packed form's flagged stream, in the FP32 pair layout, from
// the FP64-precomputed rows (M row i, b_i) of Gaussian-order table entry
// aidx[gid]; padding entries are zero.
__global__ void k_build_flag_pairs(const uint32_t* __restrict__ gid, uint32_t n, const uint32_t* __restrict__ aidx,
                                   const float4* __restrict__ table, float4* __restrict__ pairs) {
  const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= (size_t)n / 2) return;
  const uint32_t g0 = __ldg(gid + 2 * p), g1 = __ldg(gid + 2 * p + 1);
  const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float4 a = g0 == kPadGid ? z : __ldg(table + 3ull * __ldg(aidx + g0) + i);
    const float4 b = g1 == kPadGid ? z : __ldg(table + 3ull * __ldg(aidx + g1) + i);
    pairs[6 * p + 2 * i] = make_float4(a.x, b.x, a.y, b.y);
    pairs[6 * p + 2 * i + 1] = make_float4(a.z, b.z, a.w, b.w);
  }
}

// Pair p of the FP32 leaf records: entries 2p and 2p+1, rows of M and b
// interleaved lo/hi; a padding entry gets M = 0 and b = (1, 0, 0) (the plain
// form's filter discards it by its negative tolerance against |ng|^2 = 1).
__global__ void k_build_pairs(const uint32_t* __restrict__ gid, uint32_t n, const float4* __restrict__ test,
                              float4* __restrict__ pairs) {
  const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= (size_t)n / 2) return;
  const uint32_t g0 = __ldg(gid + 2 * p), g1 = __ldg(gid + 2 * p + 1);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float4 pad = make_float4(0.f, 0.f, 0.f, i == 0 ? 1.f : 0.f);
    const float4 a = g0 == kPadGid ? pad : __ldg(test + 3ull * g0 + i);
    const float4 b = g1 == kPadGid ? pad : __ldg(test + 3ull * g1 + i);
    pairs[6 * p + 2 * i] = make_float4(a.x, b.x, a.y, b.y);
    pairs[6 * p + 2 * i + 1] = make_float4(a.z, b.z, a.w, b.w);
  }
}

// The plain form's tolerance constants of pair p (Ce and Cmu, lo/hi).
__global__ void k_build_tol(const uint32_t* __restrict__ gid, uint32_t n, const float2* __restrict__ tol,
                            float4* __restrict__ out) {
  const size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= (size_t)n / 2) return;
  const uint32_t g0 = __ldg(gid + 2 * p), g1 = __ldg(gid + 2 * p + 1);
  const float2 pad = make_float2(-1.f, 0.f);
  const float2 a = g0 == kPadGid ? pad : __ldg(tol + g0), b = g1 == kPadGid ? pad : __ldg(tol + g1);
  out[p] = make_float4(a.x, b.x, a.y, b.y);
}

cudaError_t build_leaf_tol(const uint32_t* d_gid, uint32_t n_entries, const float2* tol, float4* out,
                           cudaStream_t st) {
  if (n_entries == 0) return cudaSuccess;
  const size_t np = (size_t)n_entries / 2;
  k_build_tol<<<(unsigned)((np + 255) / 256), 256, 0, st>>>(d_gid, n_entries, tol, out);
  return cudaGetLastError();
}

cudaError_t build_leaf_pairs(const uint32_t* d_gid, uint32_t n_entries, const float4* test, float4* pairs,
                             cudaStream_t st) {
  if (n_entries == 0) return cudaSuccess;
  const size_t np = (size_t)n_entries / 2;
  k_build_pairs<<<(unsigned)((np + 255) / 256), 256, 0, st>>>(d_gid, n_entries, test, pairs);
  return cudaGetLastError();
}

cudaError_t build_packed_pairs(const uint32_t* d_gid, uint32_t n_entries, const uint32_t* src, uint4* pairs,
                               cudaStream_t st) {
  if (n_entries == 0) return cudaSuccess;
  const size_t np = (size_t)n_entries / 2;
  k_build_ppairs<<<(unsigned)((np + 255) / 256), 256, 0, st>>>(d_gid, n_entries, src, pairs);
  return cudaGetLastError();
}

cudaError_t build_flag_pairs(const uint32_t* d_gid, uint32_t n_entries, const uint32_t* aidx, const float4* table,
                             float4* pairs, cudaStream_t st) {
  if (n_entries == 0) return cudaSuccess;
  const size_t np = (size_t)n_entries / 2;
  k_build_flag_pairs<<<(unsigned)((np + 255) / 256), 256, 0, st>>>(d_gid, n_entries, aidx, table, pairs);
  return cudaGetLastError();
}

cudaError_t launch_aniso_fp64(const float* src, uint32_t n, float4* table, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  k_aniso_fp64<<<(n + 127) / 128, 128, 0, st>>>(src, n, table);
  return cudaGetLastError();
}

int batch_sms() { return num_sms(); }

namespace {
constexpr int kStageViews = 256;
struct ViewStage {
  ViewDesc views[kStageViews];
  int32_t n_views;
};
static_assert(sizeof(ViewStage) <= 32764, "kernel parameters are limited to 32,764 bytes");
static_assert(kQueueBytes / sizeof(uint32_t) <= 256, "queue words are zeroed by one 256-thread block");

__global__ void __launch_bounds__(256) k_stage_views(const __grid_constant__ ViewStage p, ViewDesc* table,
                                                     uint32_t* queue) {
  const int i = threadIdx.x;
  if (i < p.n_views) table[i] = p.views[i];
  if (i < (int)(kQueueBytes / sizeof(uint32_t))) queue[i] = 0u;
}
}  // namespace

cudaError_t stage_views(const ViewDesc* views, int n_views, ViewDesc* d_views, uint32_t* d_queue, cudaStream_t st) {
  if (n_views < 0) return cudaErrorInvalidValue;
  if (n_views > kStageViews) {
    cudaError_t e = cudaMemcpyAsync(d_views, views, (size_t)n_views * sizeof(ViewDesc), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_queue, 0, kQueueBytes, st);
    return e;
  }
  ViewStage p;
  p.n_views = n_views;
  std::memcpy(p.views, views, (size_t)n_views * sizeof(ViewDesc));
  k_stage_views<<<1, 256, 0, st>>>(p, d_views, d_queue);
  return cudaGetLastError();
}

cudaError_t launch_multi(const SceneTable& scenes, bool packed, const ViewDesc* d_views, int n_views,
                         uint32_t total_blocks, uint32_t total_groups, float* const* d_outs, uint32_t* queue,
                         uint32_t* status, cudaStream_t st) {
  // The walk by the number of rays, as choose_walk (the scenes may differ), but
  // independent rays only below 100k: other lanes' launches fill the chip, and
  // packets take less of it (12 requests of 400x300: 1.86 to 2.05 ms, 1.95 to
  // 2.10 with independent rays; 8 of 300x220: 1.04 to 1.28, 0.84 to 1.05).
  const uint64_t rays = (uint64_t)kBlockW * kBlockH * total_blocks;
  const uint32_t lpr = rays < kFewRays ? 8 : 1;
  auto fn = packed ? k_render_multi<true, 8, true, 1> : k_render_multi<false, 8, true, 1>;
  if (lpr == 8) fn = packed ? k_render_multi<true, 6, true, 8> : k_render_multi<false, 6, true, 8>;
  else if (rays < 100000) fn = packed ? k_render_multi<true, 6, false, 1> : k_render_multi<false, 6, false, 1>;
  int occ = 0;
  cudaError_t e = resident_ctas(reinterpret_cast<const void*>(fn), &occ);
  if (e != cudaSuccess) return e;
  if (total_blocks > 0x3FFFFFFFu) return cudaErrorInvalidValue;
  const GroupShape gs = group_shape(4ull * total_blocks);
  const int sms = std::min(num_sms(), kMaxStrips);
  const uint32_t total = lpr == 8 ? 4u * lpr * total_blocks : total_groups;
  const int share = lpr == 8 ? sms : group_arg(sms, gs);
  uint64_t blocks = (uint64_t)num_sms() * (occ > 0 ? occ : 1);
  const uint64_t cap = (uint64_t)lpr * total_blocks;  // four items to a block, four warps to a CTA
  if (blocks > cap) blocks = cap > 0 ? cap : 1;
  fn<<<(unsigned)blocks, kThreads, 0, st>>>(scenes, d_views, n_views, total, d_outs, queue, status, share);
  return cudaGetLastError();
}

}  // namespace kdgr
