// kdbuild_gpu.cu -- the kd-tree builder on the GPU.
//
// Builds the same tree, bit for bit, as the host builder (kdbuild.cpp),
// which itself reproduces the reference builder (Kd-treeConstructor.cpp,
// PRIMITIVE_TYPE 2 / COUNT_BY_GID 1): proxy icosahedra per Gaussian
// (Kd-treeConverterMain.cpp:1860-2095), SAH split search over every distinct
// triangle-edge position with per-Gaussian-ID counting (try_to_split,
// Kd-treeConstructor.cpp:579-868), partition and clip (:364-486, :545-577),
// leaves holding their sorted unique Gaussian IDs (:1543-1549).
//
// The host builder recurses depth first; here the tree grows breadth first,
// one level per step, every node of the level at once:
//   1. runs of equal Gaussian ID inside each node (triangles stay sorted by
//      node, then ID, through every partition) give per-ID intervals
//      [mn, mx] on each axis;
//   2. the split search scores the interval ends ("events") first.  Between
//      two neighbouring events every count is constant, so the SAH cost is
//      linear in the position there and bounded below by its value at the
//      two ends: triangle edges inside a gap are scored only when that bound
//      does not exceed the best event (the tightest interval of such gaps is
//      kept per axis).  Scores are first taken in FP32; only candidates
//      within kMargin of the best FP32 score are scored in the host builder's
//      types and operation order (double costs, float extents), and the
//      smallest (cost, axis, position) wins, as in the sequential sweep.
//      Nodes of up to 1024 IDs are searched by one warp or one block each,
//      sorted interval ends in shared memory; larger nodes (the top levels)
//      by kernels over globally sorted 64-bit (axis, node, position) keys;
//   3. triangles are partitioned stably into the children (one exclusive scan
//      of packed left/right counts gives every triangle its slots) and
//      straddling ones are clipped with the host's float arithmetic, their
//      vertices recomputed from the Gaussian (a triangle is carried as its
//      clipped box, its number and its node: 32 bytes);
//   4. leaves write the IDs of their runs into one pool.
// The nodes are then numbered on the device as the reference allocates them
// (child pairs in depth-first, left-first order; leaf ID lists in the same
// order) from subtree sums taken bottom up and ranks handed down.
//
// What bounds it and why this shape: scoring every distinct edge, as the
// sequential sweep does, took a global 64-bit radix sort of all edges per
// level and about 60 FP64 operations per edge on a chip with two FP64 lanes
// per SM; events are 3 to 20 times fewer than edges, and FP64 is left for a
// handful of candidates per node -- for none where a single position is left.
// Measured on a GB300, whole call: 10k Gaussians 15.5 -> 4.0 ms, 500k 337 ->
// 61 ms, 1M 723 -> 134 ms.  Of the 500k build's 49 ms of kernels the partition
// takes 11 (3.4 TB/s), the searches 15, the scans 7, the sorts of large nodes
// 4; small builds are bound by their levels' launches and latencies.
//
// This unit is compiled with --fmad=false and IEEE division, so every float
// and double expression rounds as on the host (compiled -ffp-contract=off).
// The per-Gaussian proxy scale k_iso (a logf) is computed on the host by the
// host builder's own function, so no device math library result enters the
// tree.  Known difference: the scene box is a min/max reduction, so a box
// face exactly at -0 versus +0 may take the other zero's bits than the
// sequential host loop would.
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include <cfloat>
#include <cstdio>
#include <cstdlib>
#include <chrono>
#include <cstdint>
#include <cstring>
#include <new>
#include <string>
#include <system_error>
#include <thread>
#include <vector>

#include <unistd.h>

#include "device_pool.h"
#include "kdgr.h"
#include "kdgr_internal.h"

namespace kdgr {
namespace {

constexpr float kTravCost = 1.0f;    // TRAVL_COST
constexpr float kEmptyBonus = 0.9f;  // EMTPY_BONUS
constexpr unsigned kMinPrim = 16;    // MIN_TRI
constexpr float kEps = 0.00001f;     // KD_TREE_EPSILON
constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kFaces = 20;      // triangles per proxy: triangle t belongs to Gaussian t / kFaces

// Relative slack between FP32 and FP64 scores.  Every term of a score is
// positive (costs and extents; other parameters switch the FP32 filter off),
// so an FP32 score, at most 16 roundings from the same float inputs, is within
// 1e-6 of the FP64 one: a candidate that is not worse than the best in FP64 is
// at most 2e-6 above it in FP32.  Twice that is allowed.
constexpr float kMargin = 4e-6f;
// That needs products clear of the denormals: a node of half surface area A
// and N IDs takes an error of up to N * 2^-149 / A, below 1e-7 for any N that
// fits 32 bits of triangles when A is at least this.
constexpr float kThinArea = 1e-28f;

struct Params {
  int max_level;
  int force_split;
  float isect_cost;
  int sah_mode;
  float sort_cost;
  int filter;  // FP32 scores may discard candidates (no negative or NaN cost parameter)
};

// ------------------------------------------------------------ device buffers
// Work memory comes from the library's pool of the device (device_pool.h): it
// keeps what it has mapped while a build runs, where the device's default
// pool hands memory back at every synchronisation of the level loop.  The
// stream and the entry into the pool end with the object, on every way out.
struct Stream {
  cudaStream_t s = nullptr;
  cudaMemPool_t pool = nullptr;
  int dev = -1;
  cudaError_t err = cudaSuccess;
  Stream() {
    check(cudaGetDevice(&dev));
    if (err == cudaSuccess) check(work_pool_enter(dev, &pool));
    if (err == cudaSuccess) check(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
  }
  ~Stream() {
    if (s) {
      cudaStreamSynchronize(s);
      cudaStreamDestroy(s);
    }
    if (pool) work_pool_leave(dev);
  }
  Stream(const Stream&) = delete;
  Stream& operator=(const Stream&) = delete;
  void check(cudaError_t e) {
    if (err == cudaSuccess && e != cudaSuccess) err = e;
  }
};

template <typename T>
struct DBuf {
  T* p = nullptr;
  size_t n = 0;
  Stream* st = nullptr;
  DBuf() = default;
  DBuf(Stream& s, size_t count) { alloc(s, count); }
  void alloc(Stream& s, size_t count) {
    release();
    st = &s;
    n = count;
    if (count) st->check(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&p), count * sizeof(T), st->pool, st->s));
  }
  // at least `count` elements; the contents are not kept
  void reserve(Stream& s, size_t count) {
    if (count > n) alloc(s, count);
  }
  void release() {
    if (p && st) cudaFreeAsync(p, st->s);
    p = nullptr;
    n = 0;
  }
  void zero() {
    if (p) st->check(cudaMemsetAsync(p, 0, n * sizeof(T), st->s));
  }
  void fill_ff() {
    if (p) st->check(cudaMemsetAsync(p, 0xFF, n * sizeof(T), st->s));
  }
  ~DBuf() { release(); }
  DBuf(const DBuf&) = delete;
  DBuf& operator=(const DBuf&) = delete;
  DBuf(DBuf&& o) noexcept : p(o.p), n(o.n), st(o.st) { o.p = nullptr; o.n = 0; }
  DBuf& operator=(DBuf&& o) noexcept {
    if (this != &o) {
      release();
      p = o.p;
      n = o.n;
      st = o.st;
      o.p = nullptr;
      o.n = 0;
    }
    return *this;
  }
};

// Triangles of one level, SoA: lo/hi[a*cap + t] for the clipped box, the
// triangle's number (kFaces * valid Gaussian + face) and its node.
struct TriSet {
  DBuf<float> lo, hi;
  DBuf<uint32_t> tri, node;
  size_t cap = 0;
  void alloc(Stream& s, size_t c) {
    cap = c;
    lo.alloc(s, 3 * c);
    hi.alloc(s, 3 * c);
    tri.alloc(s, c);
    node.alloc(s, c);
  }
};
struct TriView {
  const float *lo, *hi;
  const uint32_t *tri, *node;
  size_t cap;
};
TriView view(const TriSet& t) { return TriView{t.lo.p, t.hi.p, t.tri.p, t.node.p, t.cap}; }

template <typename It, typename T>
void exclusive_sum(Stream& s, DBuf<uint8_t>& tmp, It in, T* out, size_t n) {
  if (n == 0) return;
  size_t bytes = 0;
  s.check(cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, (int64_t)n, s.s));
  tmp.reserve(s, bytes);
  s.check(cub::DeviceScan::ExclusiveSum(tmp.p, bytes, in, out, (int64_t)n, s.s));
}
// exclusive sum of op(0), op(1), ... op(n - 1), evaluated inside the scan
template <typename Op, typename T>
void exclusive_sum_of(Stream& s, DBuf<uint8_t>& tmp, Op op, T* out, size_t n) {
  exclusive_sum(s, tmp, thrust::make_transform_iterator(thrust::counting_iterator<uint64_t>(0), op), out, n);
}

void sort_keys(Stream& s, DBuf<uint8_t>& tmp, DBuf<uint64_t>& keys, DBuf<uint64_t>& alt, size_t n, int end_bit) {
  if (n == 0) return;
  cub::DoubleBuffer<uint64_t> db(keys.p, alt.p);
  size_t bytes = 0;
  s.check(cub::DeviceRadixSort::SortKeys(nullptr, bytes, db, (int64_t)n, 0, end_bit, s.s));
  tmp.reserve(s, bytes);
  s.check(cub::DeviceRadixSort::SortKeys(tmp.p, bytes, db, (int64_t)n, 0, end_bit, s.s));
  if (db.Current() != keys.p) std::swap(keys.p, alt.p);
}

// at least one block: every kernel checks its own bounds
inline unsigned grid_for(size_t n, unsigned block) { return (unsigned)std::max<size_t>(1, (n + block - 1) / block); }

// ------------------------------------------------------------ positions
// A float's bits mapped to an unsigned that sorts like the float (-0 before
// +0 as distinct keys, like the host radix sort).
__device__ __forceinline__ uint32_t ordf(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unordf(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}
// The same with -0 taken as +0: unsigned comparison of these keys is the
// float comparison.
__device__ __forceinline__ uint32_t ordz(float f) { return ordf(__fadd_rn(f, 0.0f)); }
constexpr uint32_t kZeroKey = 0x80000000u;  // ordz of either zero

// Sorted keys k[0..n): how many are < x, how many are <= x.
template <typename K>
__device__ __forceinline__ uint32_t lower(const K* k, uint32_t n, K x) {
  uint32_t lo = 0;
  while (n > 0) {
    const uint32_t h = n >> 1;
    if (k[lo + h] < x) {
      lo += h + 1;
      n -= h + 1;
    } else {
      n = h;
    }
  }
  return lo;
}
template <typename K>
__device__ __forceinline__ uint32_t upper(const K* k, uint32_t n, K x) {
  uint32_t lo = 0;
  while (n > 0) {
    const uint32_t h = n >> 1;
    if (k[lo + h] <= x) {
      lo += h + 1;
      n -= h + 1;
    } else {
      n = h;
    }
  }
  return lo;
}

__device__ __forceinline__ float ref_min(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float ref_max(float a, float b) { return a > b ? a : b; }

// ------------------------------------------------------------ proxy mesh
__constant__ float c_ico_v[12][3];
__constant__ int c_ico_f[20][3];

__device__ __forceinline__ void cross3(const float* a, const float* b, float* o) {
  o[0] = ((a[1] * b[2]) - (a[2] * b[1]));
  o[1] = -((a[0] * b[2]) - (a[2] * b[0]));
  o[2] = ((a[0] * b[1]) - (a[1] * b[0]));
}

// Vertices of proxy triangle `tri`: the icosahedron face scaled by k_iso *
// scale, rotated by the quaternion, moved to the mean (the host builder's
// proxy_icosahedron, operation for operation).  g: 10 floats per valid
// Gaussian (pos, scale, quaternion w,x,y,z).
__device__ __forceinline__ void proxy_triangle(const float* __restrict__ g, const float* __restrict__ kiso,
                                               uint32_t tri, float out[3][3]) {
  const uint32_t j = tri / kFaces, f = tri % kFaces;
  const float* gj = g + 10ull * j;
  const float k = kiso[j];
  const float fs[3] = {gj[3] * k, gj[4] * k, gj[5] * k};
  const float q0 = gj[6];
  const float qv[3] = {gj[7], gj[8], gj[9]};
#pragma unroll
  for (int l = 0; l < 3; ++l) {
    const float* vc = c_ico_v[c_ico_f[f][l]];
    const float vs[3] = {vc[0] * fs[0], vc[1] * fs[1], vc[2] * fs[2]};
    float tv[3], tt[3];
    cross3(qv, vs, tv);
#pragma unroll
    for (int i = 0; i < 3; ++i) tv[i] *= 2.0f;
    cross3(qv, tv, tt);
#pragma unroll
    for (int i = 0; i < 3; ++i) out[l][i] = (vs[i] + q0 * tv[i] + tt[i]) + gj[i];
  }
}

__global__ void k_proxy(const float* __restrict__ g, const float* __restrict__ kiso, uint32_t n_valid, float* lo,
                        float* hi, uint32_t* tri, uint32_t* node, size_t cap) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (size_t)n_valid * kFaces) return;
  float v[3][3];
  proxy_triangle(g, kiso, (uint32_t)t, v);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    lo[d * cap + t] = ref_min(ref_min(v[0][d], v[1][d]), v[2][d]);
    hi[d * cap + t] = ref_max(ref_max(v[0][d], v[1][d]), v[2][d]);
  }
  tri[t] = (uint32_t)t;
  node[t] = 0;
}

// Scene box over every proxy triangle: per-warp reduction of order-mapped
// keys, then one atomic per warp and bound.
__global__ void k_scene_box(TriView V, size_t n, uint32_t* box) {
  uint32_t mn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, mx[3] = {0, 0, 0};
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x)
    for (int d = 0; d < 3; ++d) {
      mn[d] = min(mn[d], ordf(V.lo[d * V.cap + t]));
      mx[d] = max(mx[d], ordf(V.hi[d * V.cap + t]));
    }
  for (int d = 0; d < 3; ++d) {
    const uint32_t a = __reduce_min_sync(0xFFFFFFFFu, mn[d]), b = __reduce_max_sync(0xFFFFFFFFu, mx[d]);
    if ((threadIdx.x & 31) == 0) {
      atomicMin(&box[2 * d], a);
      atomicMax(&box[2 * d + 1], b);
    }
  }
}

__global__ void k_box_decode(const uint32_t* box, float* node_lo, float* node_hi) {
  if (threadIdx.x < 3) {
    node_lo[threadIdx.x] = unordf(box[2 * threadIdx.x]);
    node_hi[threadIdx.x] = unordf(box[2 * threadIdx.x + 1]);
  }
}

// ------------------------------------------------------------ runs and nodes
// Counters of one level: nodes listed for the 128- and 512-thread searches,
// planar keys and scored candidates of the large nodes' search.
enum { kCntMid, kCntBlock, kCntPlanar, kCntScored, kCounts };

// Sizes of the next level, read back once per level.
struct LevelSum {
  unsigned long long triangles;
  uint32_t n_split, leaf_ids, max_ids;  // max_ids: most IDs in a split node
};

struct HeadOp {  // 1 where a (node, Gaussian) run starts
  const uint32_t *tri, *node;
  uint64_t T;
  __device__ uint32_t operator()(uint64_t t) const {
    if (t >= T) return 0u;
    return (t == 0 || tri[t] / kFaces != tri[t - 1] / kFaces || node[t] != node[t - 1]) ? 1u : 0u;
  }
};

// (Zeroes the level's counters as well: a memset each was a launch each.)
__global__ void k_run_scatter(const uint32_t* __restrict__ ridx, const uint32_t* __restrict__ node, size_t T,
                              uint32_t* run_start, uint32_t* run_node, uint32_t* counts, LevelSum* sum) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0) {
    for (int k = 0; k < kCounts; ++k) counts[k] = 0u;
    *sum = LevelSum{0ull, 0u, 0u, 0u};
  }
  if (t >= T) return;
  const uint32_t r = ridx[t];
  if (ridx[t + 1] == r) return;
  run_start[r] = (uint32_t)t;
  run_node[r] = node[t];
}

struct Decision {
  int axis;  // -1: leaf
  float split;
  int side;
};

// Search classes by the number of distinct IDs of a node: a warp's six lists
// of up to 64 keys sort in 21 bitonic steps and four nodes share a block's
// static shared memory; up to 256 a 128-thread block holds 21 KB, up to 1024
// a 512-thread block 86 KB, two per SM; beyond that a node alone keeps many
// blocks busy and its keys go through the device-wide sort.
constexpr uint32_t kWarpIds = 64, kMidIds = 256, kBlockIds = 1024;
// A level of few nodes takes as long as its slowest node: below this many
// nodes every one gets a 128-thread block (10k Gaussians: a warp took up to
// 130 us for a node of 64 IDs).
constexpr uint32_t kFewNodes = 4096;

// Per node: its first run, its ID count, the class lists of its split search
// (nodes of up to kWarpIds need no list) and a leaf decision to begin with.
// eG (levels that may hold larger nodes): their ID counts, 0 for the others.
__global__ void k_node_setup(const uint32_t* __restrict__ tb, const uint32_t* __restrict__ ridx, uint32_t N,
                             int level, int max_level, uint32_t warp_ids, uint32_t* rb, Decision* dec, uint32_t* is_split,
                             uint32_t* list_mid, uint32_t* list_block, uint32_t* counts, uint32_t* eG) {
  const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n > N) return;
  rb[n] = ridx[tb[n]];
  if (n == N) {
    is_split[n] = 0u;
    if (eG) eG[n] = 0u;
    return;
  }
  const uint32_t G = ridx[tb[n + 1]] - ridx[tb[n]];
  dec[n] = Decision{-1, 0.f, 0};
  is_split[n] = 0u;
  const bool elig = level < max_level && G > kMinPrim;
  if (elig && G > warp_ids && G <= kMidIds) list_mid[atomicAdd(&counts[kCntMid], 1u)] = n;
  if (elig && G > kMidIds && G <= kBlockIds) list_block[atomicAdd(&counts[kCntBlock], 1u)] = n;
  if (eG) eG[n] = elig && G > kBlockIds ? G : 0u;
}

// ------------------------------------------------------------ scores
// A node's constants of try_to_split: float extents, and in float and double
// what the scores multiply with.
struct Cell {
  float lo[3], hi[3], am[3], aa[3], rcp, init;
  uint32_t G;
};

__device__ __forceinline__ double init_cost(const Params& P, uint32_t G, uint32_t T) {
  double cost = double((size_t)G) * P.isect_cost;
  if (P.sah_mode == 7) cost = cost + P.sort_cost * (size_t)G * (size_t)G;
  if (P.force_split && (size_t)T > (size_t)P.force_split) cost = DBL_MAX;
  return cost;
}

__device__ __forceinline__ Cell make_cell(const Params& P, const float* __restrict__ nlo,
                                          const float* __restrict__ nhi, uint32_t n, uint32_t G, uint32_t T) {
  Cell c;
  float ext[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    c.lo[d] = nlo[3ull * n + d];
    c.hi[d] = nhi[3ull * n + d];
    ext[d] = c.hi[d] - c.lo[d];
  }
  const float area = (ext[0] * ext[1]) + (ext[1] * ext[2]) + (ext[0] * ext[2]);
  // below kThinArea the FP32 products round on the denormals' grid, outside
  // kMargin: NaN scores discard nothing, FP64 decides
  c.rcp = area < kThinArea ? __int_as_float(0x7fc00000) : 1.0f / area;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    c.am[a] = ext[(a + 1) % 3] + ext[(a + 2) % 3];
    c.aa[a] = ext[(a + 1) % 3] * ext[(a + 2) % 3];
  }
  c.init = __double2float_ru(init_cost(P, G, T));  // +inf for DBL_MAX
  c.G = G;
  return c;
}
template <typename V>
__device__ __forceinline__ V pick(const V v[3], int a) {
  return a == 0 ? v[0] : a == 1 ? v[1] : v[2];
}

__device__ __forceinline__ bool in_limits(const Cell& c, int a, float p) {
  return p > pick(c.lo, a) + kEps && p < pick(c.hi, a) - kEps;
}

// Counts at a position: intervals begun before it, ended before it, ended at
// it, and planar at it.
struct Counts {
  uint32_t open, close, eq_max, planar;
};

// FP32 score (the better of the two planar sides).
__device__ __forceinline__ float score32(const Params& P, const Cell& c, int a, float p, const Counts& k) {
  const float pl = ((p - pick(c.lo, a)) * pick(c.am, a) + pick(c.aa, a)) * c.rcp;
  const float pr = ((pick(c.hi, a) - p) * pick(c.am, a) + pick(c.aa, a)) * c.rcp;
  const int tl1 = (int)k.open, tr0 = (int)(c.G - k.close - k.eq_max), pn = (int)k.planar;
  float best = __int_as_float(0x7f800000);
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    if (s == 1 && pn == 0) break;  // both sides score the same
    const int il = s == 0 ? tl1 + pn : tl1, ir = s == 0 ? tr0 : tr0 + pn;
    const float tl = (float)il, tr = (float)ir;
    const float eb = (il == 0 || ir == 0) ? kEmptyBonus : 1.0f;
    float v;
    if (P.sah_mode == 4) {
      v = kTravCost + P.isect_cost * (tl * sqrtf(tl * 0.0625f) * pl + tr * sqrtf(tr * 0.0625f) * pr) * eb;
    } else {
      v = P.isect_cost * (tl * pl + tr * pr) * eb;
      if (P.sah_mode != 0 && P.sah_mode != 7) v *= 1.0f + __fdividef(fabsf(tl - tr), fmaxf(tl + tr, 1.0f)) * 0.1f;
      v += kTravCost;
      if (P.sah_mode == 7) v += P.sort_cost * (tl * tl * pl + tr * tr * pr);
    }
    if (!(v < __int_as_float(0x7f800000))) return __int_as_float(0x7fc00000);  // overflow: NaN, never discarded
    best = v < best ? v : best;
  }
  return best;
}

// The host builder's score, its types and operation order.
__device__ __noinline__ double score64(const Params& P, const float* __restrict__ nlo, const float* __restrict__ nhi,
                                       uint32_t n, uint32_t G, int a, float p, Counts k, int* side) {
  float ext[3];
  for (int d = 0; d < 3; ++d) ext[d] = nhi[3ull * n + d] - nlo[3ull * n + d];
  const float cell_area_f = (ext[0] * ext[1]) + (ext[1] * ext[2]) + (ext[0] * ext[2]);
  const double cell_area = cell_area_f;
  const double cell_area_rcp = 1 / cell_area;
  const int a1 = (a + 1) % 3, a2 = (a + 2) % 3;
  const double area_mul = double(pick(ext, a1)) + double(pick(ext, a2));
  const double area_add = double(pick(ext, a1)) * double(pick(ext, a2));
  const float cell_min = nlo[3ull * n + a], cell_max = nhi[3ull * n + a];
  const int num_planars = (int)k.planar;
  const int local_close = (int)k.eq_max - num_planars;
  const double extent_l = double(p) - cell_min;
  const double extent_r = cell_max - double(p);
  const double prob_l = (extent_l * area_mul + area_add) * cell_area_rcp;
  const double prob_r = (extent_r * area_mul + area_add) * cell_area_rcp;
  const int n_left_only = (int)k.close + local_close;
  const int n_cross = (int)k.open - n_left_only;
  const int n_right_only = int(G) - (n_left_only + n_cross + num_planars);
  const int tl[2] = {n_left_only + n_cross + num_planars, n_left_only + n_cross};
  const int tr[2] = {n_right_only + n_cross, n_right_only + n_cross + num_planars};
  const float eb[2] = {(tl[0] == 0 || tr[0] == 0) ? kEmptyBonus : 1.0f,
                       (tl[1] == 0 || tr[1] == 0) ? kEmptyBonus : 1.0f};
  double sah[2];
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    switch (P.sah_mode) {
      case 0:
        sah[s] = kTravCost + P.isect_cost * (double(tl[s]) * prob_l + double(tr[s]) * prob_r) * eb[s];
        break;
      case 4: {
        // n * pow(n / 16, 0.5) with the square root, which is what a
        // correctly rounded pow returns for the exponent 0.5
        const double xl = double(tl[s]), xr = double(tr[s]);
        const double sl = tl[s] == 0 ? 0.0 : xl * sqrt(xl / 16.0);
        const double sr = tr[s] == 0 ? 0.0 : xr * sqrt(xr / 16.0);
        sah[s] = kTravCost + P.isect_cost * (sl * prob_l + sr * prob_r) * eb[s];
        break;
      }
      case 7:
        sah[s] = kTravCost + P.isect_cost * (double(tl[s]) * prob_l + double(tr[s]) * prob_r) * eb[s] +
                 P.sort_cost * (double(tl[s]) * double(tl[s]) * prob_l + double(tr[s]) * double(tr[s]) * prob_r);
        break;
      default: {
        const double n_total = double(tl[s] + tr[s]);
        const double diff = fabs(double(tl[s]) - double(tr[s]));
        const double ratio = (n_total > 0.0) ? (diff / n_total) : 0.0;
        const double penalty = 1.0 + (ratio * 0.1);
        sah[s] = kTravCost + P.isect_cost * (double(tl[s]) * prob_l + double(tr[s]) * prob_r) * eb[s] * penalty;
        break;
      }
    }
  }
  *side = sah[0] <= sah[1] ? 0 : 1;
  return sah[0] <= sah[1] ? sah[0] : sah[1];
}

// Candidates in the sequential sweep's order: lowest axis, then lowest
// position (bits), the planar side riding along.
__device__ __forceinline__ uint64_t cand_key(int a, float p, int side) {
  return ((uint64_t)a << 33) | ((uint64_t)ordf(p) << 1) | (uint64_t)side;
}
__device__ __forceinline__ Decision key_decision(uint64_t k) {
  return Decision{(int)(k >> 33), unordf((uint32_t)(k >> 1)), (int)(k & 1u)};
}

// ------------------------------------------------------------ split search of one node
// NT threads (a warp or a block) search one node of at most CAP IDs.  Per
// axis the interval starts and ends are sorted in shared memory (bitonic;
// 6 lists side by side), every event is scored in FP32 with its gap bound,
// the few candidates within the margin are scored in FP64, then the node's
// triangle edges inside the surviving gaps.
template <int NT, int CAP>
struct SearchMem {
  uint32_t k[6][CAP];       // sorted ordz keys: starts of axes 0..2, ends of axes 0..2
  uint32_t pl[3][CAP];      // planar positions, unsorted
  float cost[6][CAP], bound[6][CAP];
  uint32_t n_pl[3], hull_lo[3], hull_hi[3];
  uint64_t cand[CAP];       // candidates within the margin: axis << 32 | ordf(position)
  uint32_t n_cand;
  float red[NT / 32];
  double best_c[NT / 32];
  uint64_t best_k[NT / 32];
};

template <int NT>
__device__ __forceinline__ void group_sync() {
  if (NT == 32) __syncwarp();
  else __syncthreads();
}

// tid: index inside the group.  n: node; runs [r0, r0 + G), triangles [t0, t1); ridx[t + 1] - 1: run of triangle t.
template <int NT, int CAP>
__device__ __forceinline__ void search_node(SearchMem<NT, CAP>& S, int tid, const Params& P, uint32_t n, uint32_t r0,
                                            uint32_t G, uint32_t t0, uint32_t t1,
                                            const uint32_t* __restrict__ ridx, const TriView& V,
                                            const float* __restrict__ nlo, const float* __restrict__ nhi,
                                            Decision* dec, uint32_t* is_split) {
  const float kInf = __int_as_float(0x7f800000);
  uint32_t M = 32, shift = 5;
  while (M < G) {
    M <<= 1;
    ++shift;
  }
  if (tid == 0) S.n_cand = 0u;
  if (tid < 3) {
    S.n_pl[tid] = 0u;
    S.hull_lo[tid] = 0xFFFFFFFFu;
    S.hull_hi[tid] = 0u;
  }
  group_sync<NT>();
  for (uint32_t r = tid; r < M; r += NT)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      S.k[a][r] = 0xFFFFFFFFu;
      S.k[3 + a][r] = r < G ? 0u : 0xFFFFFFFFu;
    }
  group_sync<NT>();
  // Interval of every ID: a warp takes 32 triangles at a time, coalesced,
  // reduces each run's part of them by shuffles and the run's first lane
  // merges it.
  for (uint32_t b = t0 + (tid & ~31u); b < t1; b += NT) {
    const uint32_t t = b + (tid & 31u), tc = min(t, t1 - 1);
    const uint32_t r = ridx[tc + 1] - 1u - r0;
    uint32_t v[6];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      v[a] = ordz(V.lo[a * V.cap + tc]);
      v[3 + a] = ordz(V.hi[a * V.cap + tc]);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      // runs are contiguous: lane + o is in this lane's run if its index is the same
      const bool same = __shfl_down_sync(0xFFFFFFFFu, r, o) == r && (tid & 31u) + o < 32u;
#pragma unroll
      for (int l = 0; l < 6; ++l) {
        const uint32_t w = __shfl_down_sync(0xFFFFFFFFu, v[l], o);
        if (same) v[l] = l < 3 ? min(v[l], w) : max(v[l], w);
      }
    }
    const uint32_t before = __shfl_up_sync(0xFFFFFFFFu, r, 1);
    const bool head = (tid & 31u) == 0u || before != r;
    if (head && t < t1) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        atomicMin(&S.k[a][r], v[a]);
        atomicMax(&S.k[3 + a][r], v[3 + a]);
      }
    }
  }
  group_sync<NT>();
  for (uint32_t r = tid; r < G; r += NT)
#pragma unroll
    for (int a = 0; a < 3; ++a)
      if (S.k[a][r] == S.k[3 + a][r]) S.pl[a][atomicAdd(&S.n_pl[a], 1u)] = S.k[a][r];
  group_sync<NT>();
  // bitonic sort of the six lists
  for (uint32_t size = 2; size <= M; size <<= 1)
    for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
      for (uint32_t i = tid; i < 6 * (M / 2); i += NT) {
        const uint32_t l = i >> (shift - 1), j = i & (M / 2 - 1);
        const uint32_t x = 2 * j - (j & (stride - 1)), y = x + stride;
        const uint32_t u = S.k[l][x], v = S.k[l][y];
        if ((u > v) == ((x & size) == 0)) {
          S.k[l][x] = v;
          S.k[l][y] = u;
        }
      }
      group_sync<NT>();
    }
  const Cell c = make_cell(P, nlo, nhi, n, G, t1 - t0);
  auto counts_at = [&](int a, uint32_t kp) {
    Counts k;
    k.open = lower(S.k[a], G, kp);
    k.close = lower(S.k[3 + a], G, kp);
    k.eq_max = upper(S.k[3 + a], G, kp) - k.close;
    k.planar = 0;
    for (uint32_t j = 0; j < S.n_pl[a]; ++j) k.planar += S.pl[a][j] == kp ? 1u : 0u;
    return k;
  };
  // events: FP32 score, and a lower bound over the gap up to the next event
  float best32 = c.init;
  for (uint32_t i = tid; i < 6 * M; i += NT) {
    const uint32_t l = i >> shift, j = i & (M - 1);
    if (j >= G) continue;
    const int a = (int)(l < 3 ? l : l - 3);
    const uint32_t kp = S.k[l][j];
    const float p = unordf(kp);
    float cost = kInf, bound = kInf;
    if (!(j > 0 && S.k[l][j - 1] == kp)) {  // equal events score once
      // the event is the first of its value in its own list: only the other
      // list is searched
      const uint32_t* const own = S.k[l];
      const uint32_t* const other = S.k[l < 3 ? l + 3 : l - 3];
      uint32_t own_le = j + 1;
      while (own_le < G && own[own_le] == kp) ++own_le;
      const uint32_t lt = lower(other, G, kp);
      uint32_t le = lt;
      while (le < G && other[le] == kp) ++le;
      Counts k{l < 3 ? j : lt, l < 3 ? lt : j, 0u, 0u};
      const uint32_t le_mn = l < 3 ? own_le : le, le_mx = l < 3 ? le : own_le;
      k.eq_max = le_mx - k.close;
      if (in_limits(c, a, p)) {
        for (uint32_t i2 = 0; i2 < S.n_pl[a]; ++i2) k.planar += S.pl[a][i2] == kp ? 1u : 0u;
        cost = score32(P, c, a, p, k);
      }
      const uint32_t nmn = le_mn < G ? S.k[a][le_mn] : 0xFFFFFFFFu, nmx = le_mx < G ? S.k[3 + a][le_mx] : 0xFFFFFFFFu;
      const uint32_t kn = min(nmn, nmx);
      if (kn != 0xFFFFFFFFu) {
        const float q = unordf(kn);
        const float pa = fmaxf(p, pick(c.lo, a) + kEps), pb = fminf(q, pick(c.hi, a) - kEps);
        if (!(pa > pb)) {
          const Counts kg{le_mn, le_mx, 0u, 0u};
          const float ba = score32(P, c, a, pa, kg), bb = score32(P, c, a, pb, kg);
          bound = (ba < bb || !(ba == ba)) ? ba : bb;
        }
      }
    }
    S.cost[l][j] = cost;
    S.bound[l][j] = bound;
    best32 = cost < best32 ? cost : best32;
  }
  for (int o = 16; o > 0; o >>= 1) best32 = fminf(best32, __shfl_xor_sync(0xFFFFFFFFu, best32, o));
  if (NT > 32) {
    if ((tid & 31) == 0) S.red[tid >> 5] = best32;
    __syncthreads();
    for (int w = 0; w < NT / 32; ++w) best32 = fminf(best32, S.red[w]);
  }
  const float limit = P.filter ? best32 * (1.0f + kMargin) : kInf;
  const double init = init_cost(P, G, t1 - t0);
  double best = init;
  uint64_t best_k = ~0ull;
  auto consider = [&](int a, float p, const Counts& k) {
    int side;
    const double cst = score64(P, nlo, nhi, n, G, a, p, k, &side);
    if (cst < init) {
      const uint64_t key = cand_key(a, p, side);
      if (cst < best || (cst == best && key < best_k)) {
        best = cst;
        best_k = key;
      }
    }
  };
  // Candidates within the margin are gathered first and scored in FP64 side by
  // side: the SM's two FP64 lanes take some 1100 cycles for one score, whether
  // one thread of a warp or all of them ask for it.
  auto gather = [&](int a, float p) {
    const uint32_t at = atomicAdd(&S.n_cand, 1u);
    if (at < (uint32_t)CAP) S.cand[at] = (uint64_t)a << 32 | ordf(p);
  };
  // events and gaps that are not worse than the best by more than the margin
  for (uint32_t i = tid; i < 6 * M; i += NT) {
    const uint32_t l = i >> shift, j = i & (M - 1);
    if (j >= G) continue;
    const int a = (int)(l < 3 ? l : l - 3);
    const float cost = S.cost[l][j], bound = S.bound[l][j];
    if (!(cost > limit) && cost != kInf) {
      const uint32_t kp = S.k[l][j];
      gather(a, unordf(kp));
      if (kp == kZeroKey) {  // the edges at zero say which zero it is
        atomicMin(&S.hull_lo[a], kp);
        atomicMax(&S.hull_hi[a], kp);
      }
    }
    if (!(bound > limit) && (bound != kInf || !P.filter)) {
      const uint32_t kp = S.k[l][j];
      const uint32_t le_mn = upper(S.k[a], G, kp), le_mx = upper(S.k[3 + a], G, kp);
      const uint32_t kn = min(le_mn < G ? S.k[a][le_mn] : 0xFFFFFFFFu, le_mx < G ? S.k[3 + a][le_mx] : 0xFFFFFFFFu);
      atomicMin(&S.hull_lo[a], kp);
      atomicMax(&S.hull_hi[a], kn);
    }
  }
  group_sync<NT>();
  // triangle edges inside the surviving gaps (interval ends among them: their
  // own bits decide between -0 and +0)
  auto edges = [&](auto take) {
    for (int a = 0; a < 3; ++a) {
      const uint32_t hl = S.hull_lo[a], hh = S.hull_hi[a];
      if (hl > hh) continue;
      for (uint32_t t = t0 + tid; t < t1; t += NT) {
        const float e[2] = {V.lo[a * V.cap + t], V.hi[a * V.cap + t]};
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const float p = e[s];
          const uint32_t kp = ordz(p);
          if (kp < hl || kp > hh || !in_limits(c, a, p)) continue;
          const Counts k = counts_at(a, kp);
          if (score32(P, c, a, p, k) > limit) continue;
          take(a, p, k);
        }
      }
    }
  };
  edges([&](int a, float p, const Counts&) { gather(a, p); });
  group_sync<NT>();
  const uint32_t m = S.n_cand;
  if (m > 0u && m <= (uint32_t)CAP) {
    const uint64_t c0 = S.cand[0];
    const int a = (int)(c0 >> 32);
    const float p = unordf((uint32_t)c0);
    bool same = true;
    for (uint32_t i = tid; i < m; i += NT) same = same && S.cand[i] == c0;
    same = NT == 32 ? __all_sync(0xFFFFFFFFu, same) : __syncthreads_and(same);
    const Counts k0 = counts_at(a, ordz(p));
    if (P.filter && same && k0.planar == 0 && (double)score32(P, c, a, p, k0) * (1.0 + kMargin) < init) {
      // one position is left and it certainly beats the leaf: its cost decides
      // nothing more, and without planar IDs both sides score the same (the
      // margin bounds positive scores only: other costs go to FP64)
      best_k = cand_key(a, p, 0);
    } else {
      for (uint32_t i = tid; i < m; i += NT) {
        const uint64_t ci = S.cand[i];
        const int ai = (int)(ci >> 32);
        consider(ai, unordf((uint32_t)ci), counts_at(ai, ordz(unordf((uint32_t)ci))));
      }
    }
  } else if (m > (uint32_t)CAP) {  // more than the list holds (no filter, or a flat node): each on the spot
    for (uint32_t i = tid; i < 6 * M; i += NT) {
      const uint32_t l = i >> shift, j = i & (M - 1);
      if (j >= G) continue;
      const int a = (int)(l < 3 ? l : l - 3);
      const float cost = S.cost[l][j];
      if (!(cost > limit) && cost != kInf) consider(a, unordf(S.k[l][j]), counts_at(a, S.k[l][j]));
    }
    edges(consider);
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double oc = __shfl_xor_sync(0xFFFFFFFFu, best, o);
    const uint64_t ok = __shfl_xor_sync(0xFFFFFFFFu, best_k, o);
    if (oc < best || (oc == best && ok < best_k)) {
      best = oc;
      best_k = ok;
    }
  }
  if (NT > 32) {
    if ((tid & 31) == 0) {
      S.best_c[tid >> 5] = best;
      S.best_k[tid >> 5] = best_k;
    }
    __syncthreads();
    for (int w = 0; w < NT / 32; ++w)
      if (S.best_c[w] < best || (S.best_c[w] == best && S.best_k[w] < best_k)) {
        best = S.best_c[w];
        best_k = S.best_k[w];
      }
  }
  if (tid == 0 && best_k != ~0ull) {
    dec[n] = key_decision(best_k);
    is_split[n] = 1u;
  }
}

// Nodes of up to kWarpIds IDs: one warp each, over every node of the level.
constexpr int kSearchWarps = 4;
__global__ void __launch_bounds__(32 * kSearchWarps)
    k_search_warp(Params P, uint32_t N, int level, const uint32_t* __restrict__ tb, const uint32_t* __restrict__ rb,
                  const uint32_t* __restrict__ ridx, TriView V, const float* __restrict__ nlo,
                  const float* __restrict__ nhi, Decision* dec, uint32_t* is_split) {
  __shared__ SearchMem<32, kWarpIds> S[kSearchWarps];
  const int w = threadIdx.x >> 5;
  const uint32_t n = blockIdx.x * kSearchWarps + w;
  if (n >= N || level >= P.max_level) return;
  const uint32_t r0 = rb[n], G = rb[n + 1] - r0;
  if (G <= kMinPrim || G > kWarpIds) return;
  search_node<32, (int)kWarpIds>(S[w], threadIdx.x & 31, P, n, r0, G, tb[n], tb[n + 1], ridx, V, nlo, nhi, dec,
                                 is_split);
}

// Listed nodes: one block each (the grid walks the list).
template <int NT, int CAP>
__global__ void __launch_bounds__(NT)
    k_search_block(Params P, const uint32_t* __restrict__ list, const uint32_t* __restrict__ count,
                   const uint32_t* __restrict__ tb, const uint32_t* __restrict__ rb,
                   const uint32_t* __restrict__ ridx, TriView V, const float* __restrict__ nlo,
                   const float* __restrict__ nhi, Decision* dec, uint32_t* is_split) {
  extern __shared__ __align__(16) unsigned char raw[];
  SearchMem<NT, CAP>& S = *reinterpret_cast<SearchMem<NT, CAP>*>(raw);
  for (uint32_t i = blockIdx.x; i < *count; i += gridDim.x) {
    const uint32_t n = list[i], r0 = rb[n];
    search_node<NT, CAP>(S, threadIdx.x, P, n, r0, rb[n + 1] - r0, tb[n], tb[n + 1], ridx, V, nlo, nhi, dec,
                         is_split);
    __syncthreads();
  }
}

// ------------------------------------------------------------ split search of large nodes
// The same search over globally sorted keys: (axis, node, position) -> 64 bits
// ordered by axis, then node, then position (ordz).
__device__ __forceinline__ uint64_t make_key(int axis, uint32_t node, uint32_t kp, int nb) {
  return ((uint64_t)axis << (32 + nb)) | ((uint64_t)node << 32) | kp;
}
__device__ __forceinline__ void decode(uint64_t k, int nb, int* a, uint32_t* n) {
  *a = (int)(k >> (32 + nb));
  *n = (uint32_t)((k >> 32) & ((1ull << nb) - 1));
}

struct Big {
  const uint64_t *kmin, *kmax, *kpl;  // sorted keys; node n's segment on axis a starts at a * eG + grb[n]
  const uint32_t *grb, *eGn;          // first slot of each large node, its ID count (0: not large)
  size_t eG;                          // IDs of all large nodes
  uint32_t n_pl;
  int nb;
};

// Per run of a large node: the ID's interval on each axis (first triangle's
// box, then strict comparisons, in triangle order, as the host sweep builds
// it) as keys.
__global__ void k_run_bounds(const uint32_t* __restrict__ run_start, const uint32_t* __restrict__ run_node,
                             const uint32_t* __restrict__ rb, uint32_t N, size_t T, TriView V, Big B, uint64_t* kmin,
                             uint64_t* kmax, uint64_t* kpl, uint32_t* pl_fill) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= rb[N]) return;
  const uint32_t n = run_node[r];
  if (B.eGn[n] == 0u) return;
  const uint32_t t0 = run_start[r], t1 = r + 1 < rb[N] ? run_start[r + 1] : (uint32_t)T;
  const size_t slot = B.grb[n] + (r - rb[n]);
  for (int a = 0; a < 3; ++a) {
    float mn = V.lo[a * V.cap + t0], mx = V.hi[a * V.cap + t0];
    for (uint32_t t = t0 + 1; t < t1; ++t) {
      const float l = V.lo[a * V.cap + t], h = V.hi[a * V.cap + t];
      if (l < mn) mn = l;
      if (h > mx) mx = h;
    }
    kmin[a * B.eG + slot] = make_key(a, n, ordz(mn), B.nb);
    kmax[a * B.eG + slot] = make_key(a, n, ordz(mx), B.nb);
    if (mn == mx) kpl[atomicAdd(pl_fill, 1u)] = make_key(a, n, ordz(mn), B.nb);
  }
}

__device__ __forceinline__ Counts big_counts(const Big& B, int a, uint32_t n, uint32_t kp) {
  const size_t b = a * B.eG + B.grb[n];
  const uint32_t G = B.eGn[n];
  const uint64_t key = make_key(a, n, kp, B.nb);
  Counts k;
  k.open = lower(B.kmin + b, G, key);
  k.close = lower(B.kmax + b, G, key);
  k.eq_max = upper(B.kmax + b, G, key) - k.close;
  k.planar = B.n_pl ? upper(B.kpl, B.n_pl, key) - lower(B.kpl, B.n_pl, key) : 0u;
  return k;
}

// State of a large node's search: best FP32 event (float bits; scores are
// positive where the filter is on), best FP64 cost, its first candidate, and
// per axis the hull of the surviving gaps.
// The candidates scored in FP64 are listed (there are few within the margin),
// so that choosing among those of equal cost does not score them again; only
// when the list overflows (no FP32 filter) do the two scoring passes run twice.
struct Scored {
  unsigned long long cost, key;
  uint32_t node;
};
constexpr uint32_t kScoredCap = 1u << 20;
struct BigState {
  uint32_t* best32;
  unsigned long long *best64, *key;
  uint32_t *hull_lo, *hull_hi;
  Scored* list;
  uint32_t* n_list;
};
// order-preserving map of a double to unsigned
__device__ __forceinline__ unsigned long long ordd(double d) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(d);
  return (u >> 63) ? ~u : (u | 0x8000000000000000ull);
}

// Pass 1: FP32 score and gap bound of every event; the node's best score.
__global__ void k_event_scores(Params P, Big B, const uint32_t* __restrict__ tb, const float* __restrict__ nlo,
                               const float* __restrict__ nhi, float2* out, BigState st) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const float kInf = __int_as_float(0x7f800000);
  float cost = kInf, bound = kInf;
  uint32_t n = kNone;
  if (i < 6 * B.eG) {
    const bool is_max = i >= 3 * B.eG;
    const size_t j = is_max ? i - 3 * B.eG : i;
    const uint64_t* own = is_max ? B.kmax : B.kmin;
    const uint64_t key = own[j];
    int a;
    decode(key, B.nb, &a, &n);
    if (j == 0 || own[j - 1] != key) {
      const uint32_t kp = (uint32_t)key, G = B.eGn[n];
      const float p = unordf(kp);
      const Cell c = make_cell(P, nlo, nhi, n, G, tb[n + 1] - tb[n]);
      const Counts k = big_counts(B, a, n, kp);
      if (in_limits(c, a, p)) cost = score32(P, c, a, p, k);
      const size_t b = a * B.eG + B.grb[n];
      const uint32_t le_mn = upper(B.kmin + b, G, key), le_mx = k.close + k.eq_max;
      const uint32_t kn = min(le_mn < G ? (uint32_t)B.kmin[b + le_mn] : 0xFFFFFFFFu,
                              le_mx < G ? (uint32_t)B.kmax[b + le_mx] : 0xFFFFFFFFu);
      if (kn != 0xFFFFFFFFu) {
        const float pa = fmaxf(p, pick(c.lo, a) + kEps), pb = fminf(unordf(kn), pick(c.hi, a) - kEps);
        if (!(pa > pb)) {
          const Counts kg{le_mn, le_mx, 0u, 0u};
          const float ba = score32(P, c, a, pa, kg), bb = score32(P, c, a, pb, kg);
          bound = (ba < bb || !(ba == ba)) ? ba : bb;
        }
      }
    }
    out[i] = make_float2(cost, bound);
  }
  // one atomic per warp when its events belong to one node, as nearly all do
  const uint32_t bits = cost >= 0.0f ? __float_as_uint(cost) : 0x7f800000u;  // NaN and negative: no limit from them
  const uint32_t lead = __shfl_sync(0xFFFFFFFFu, n, 0);
  if (__all_sync(0xFFFFFFFFu, n == lead)) {
    const uint32_t m = __reduce_min_sync(0xFFFFFFFFu, bits);
    if ((threadIdx.x & 31) == 0 && n != kNone && m < 0x7f800000u) atomicMin(&st.best32[n], m);
  } else if (n != kNone && bits < 0x7f800000u) {
    atomicMin(&st.best32[n], bits);
  }
}

__device__ __forceinline__ float big_limit(const Params& P, const BigState& st, uint32_t n) {
  return P.filter ? __uint_as_float(st.best32[n]) * (1.0f + kMargin) : __int_as_float(0x7f800000);
}

// FIRST: reduce the FP64 cost; otherwise the first candidate that has it.
template <bool FIRST>
__device__ __forceinline__ void big_consider(const Params& P, const Big& B, const BigState& st,
                                             const uint32_t* __restrict__ tb, const float* __restrict__ nlo,
                                             const float* __restrict__ nhi, uint32_t n, int a, float p,
                                             const Counts& k) {
  int side;
  const double cst = score64(P, nlo, nhi, n, B.eGn[n], a, p, k, &side);
  if (!(cst < init_cost(P, B.eGn[n], tb[n + 1] - tb[n]))) return;
  const unsigned long long o = ordd(cst);
  if (FIRST) {
    if (o > st.best64[n]) return;  // only ever decreases
    atomicMin(&st.best64[n], o);
    const uint32_t at = atomicAdd(st.n_list, 1u);
    if (at < kScoredCap) st.list[at] = Scored{o, cand_key(a, p, side), n};
  } else if (o == st.best64[n]) {
    atomicMin(&st.key[n], (unsigned long long)cand_key(a, p, side));
  }
}

// Pass 2 (FIRST; again if the list overflowed): events within the margin; pass 2 also gathers the
// hull of the gaps whose bound is.
template <bool FIRST>
__global__ void k_event_exact(Params P, Big B, const uint32_t* __restrict__ tb, const float* __restrict__ nlo,
                              const float* __restrict__ nhi, const float2* __restrict__ scores, BigState st) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 6 * B.eG || (!FIRST && *st.n_list <= kScoredCap)) return;
  const float kInf = __int_as_float(0x7f800000);
  const bool is_max = i >= 3 * B.eG;
  const uint64_t key = is_max ? B.kmax[i - 3 * B.eG] : B.kmin[i];
  int a;
  uint32_t n;
  decode(key, B.nb, &a, &n);
  const float limit = big_limit(P, st, n);
  const float2 s = scores[i];
  const uint32_t kp = (uint32_t)key;
  if (!(s.x > limit) && s.x != kInf) {
    big_consider<FIRST>(P, B, st, tb, nlo, nhi, n, a, unordf(kp), big_counts(B, a, n, kp));
    if (FIRST && kp == kZeroKey) {  // the edges at zero say which zero it is
      atomicMin(&st.hull_lo[3ull * n + a], kp);
      atomicMax(&st.hull_hi[3ull * n + a], kp);
    }
  }
  if (FIRST && !(s.y > limit) && (s.y != kInf || !P.filter)) {
    const size_t b = a * B.eG + B.grb[n];
    const uint32_t G = B.eGn[n];
    const uint32_t le_mn = upper(B.kmin + b, G, key), le_mx = upper(B.kmax + b, G, key);
    const uint32_t kn = min(le_mn < G ? (uint32_t)B.kmin[b + le_mn] : 0xFFFFFFFFu,
                            le_mx < G ? (uint32_t)B.kmax[b + le_mx] : 0xFFFFFFFFu);
    atomicMin(&st.hull_lo[3ull * n + a], kp);
    atomicMax(&st.hull_hi[3ull * n + a], kn);
  }
}

// Pass 3 (FIRST; again if the list overflowed): triangle edges inside the hulls.
template <bool FIRST>
__global__ void k_edge_exact(Params P, Big B, TriView V, size_t T, const uint32_t* __restrict__ tb,
                             const float* __restrict__ nlo, const float* __restrict__ nhi, BigState st) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T || (!FIRST && *st.n_list <= kScoredCap)) return;
  const uint32_t n = V.node[t];
  if (B.eGn[n] == 0u) return;
  for (int a = 0; a < 3; ++a) {
    const uint32_t hl = st.hull_lo[3ull * n + a], hh = st.hull_hi[3ull * n + a];
    if (hl > hh) continue;
    const float e[2] = {V.lo[a * V.cap + t], V.hi[a * V.cap + t]};
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const float p = e[s];
      const uint32_t kp = ordz(p);
      if (kp < hl || kp > hh) continue;
      const Cell c = make_cell(P, nlo, nhi, n, B.eGn[n], tb[n + 1] - tb[n]);
      if (!in_limits(c, a, p)) continue;
      const Counts k = big_counts(B, a, n, kp);
      if (score32(P, c, a, p, k) > big_limit(P, st, n)) continue;
      big_consider<FIRST>(P, B, st, tb, nlo, nhi, n, a, p, k);
    }
  }
}

__global__ void k_big_init(const Params P, Big B, const uint32_t* __restrict__ tb, uint32_t N, BigState st) {
  const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  const float init = __double2float_ru(init_cost(P, B.eGn[n], tb[n + 1] - tb[n]));
  st.best32[n] = init >= 0.0f ? __float_as_uint(init) : 0x7f800000u;
  st.best64[n] = ~0ull;
  st.key[n] = ~0ull;
  for (int a = 0; a < 3; ++a) {
    st.hull_lo[3ull * n + a] = 0xFFFFFFFFu;
    st.hull_hi[3ull * n + a] = 0u;
  }
}

// First candidate of each node's smallest cost, from the list.
__global__ void k_scored_first(BigState st) {
  const uint32_t m = *st.n_list;
  if (m > kScoredCap) return;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    const Scored c = st.list[i];
    if (c.cost == st.best64[c.node]) atomicMin(&st.key[c.node], c.key);
  }
}

__global__ void k_big_choose(Big B, uint32_t N, BigState st, Decision* dec, uint32_t* is_split) {
  const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N || B.eGn[n] == 0u || st.key[n] == ~0ull) return;
  dec[n] = key_decision(st.key[n]);
  is_split[n] = 1u;
}

// ------------------------------------------------------------ partition
// Which children a triangle goes to (push_triangles_to_child_vector).
__device__ __forceinline__ void sides_of(float mn, float mx, const Decision& d, bool* l, bool* r) {
  if (mn != mx) {
    *l = mn < d.split;
    *r = mx > d.split;
  } else {
    *l = mn < d.split || (mn == d.split && d.side == 0);
    *r = mn > d.split || (mn == d.split && d.side != 0);
  }
}

struct SideOp {  // left count in the low word, right count in the high word
  TriView V;
  const Decision* dec;
  uint64_t T;
  __device__ uint64_t operator()(uint64_t t) const {
    if (t >= T) return 0ull;
    const Decision d = dec[V.node[t]];
    if (d.axis < 0) return 0ull;
    bool l, r;
    sides_of(V.lo[d.axis * V.cap + t], V.hi[d.axis * V.cap + t], d, &l, &r);
    return (l ? 1ull : 0ull) | (r ? 1ull << 32 : 0ull);
  }
};
__device__ __forceinline__ uint32_t lo32(uint64_t x) { return (uint32_t)x; }
__device__ __forceinline__ uint32_t hi32(uint64_t x) { return (uint32_t)(x >> 32); }

struct NodeOp {  // split nodes in the low word, leaf IDs in the high word
  const uint32_t *is_split, *rb;
  uint32_t N;
  __device__ uint64_t operator()(uint64_t n) const {
    if (n >= N) return 0ull;
    return is_split[n] ? 1ull : (uint64_t)(rb[n + 1] - rb[n]) << 32;
  }
};

// clip_triangle for one straddling triangle (host clip_tri, same arithmetic):
// where the segment p0 p1 meets the plane x[axis] = split.
__device__ __forceinline__ bool edge_plane(const float* p0, const float* p1, const float* pp, const float* pn,
                                           float* hit) {
  float u[3], w[3];
  u[0] = p1[0] - p0[0];
  u[1] = p1[1] - p0[1];
  u[2] = p1[2] - p0[2];
  w[0] = p0[0] - pp[0];
  w[1] = p0[1] - pp[1];
  w[2] = p0[2] - pp[2];
  const float D = pn[0] * u[0] + pn[1] * u[1] + pn[2] * u[2];
  const float Nn = -(pn[0] * w[0] + pn[1] * w[1] + pn[2] * w[2]);
  if (fabsf(D) < kEps) return false;
  const float sI = Nn / D;
  if (sI < 0.f || sI > 1.f) return false;
  hit[0] = p0[0] + u[0] * sI;
  hit[1] = p0[1] + u[1] * sI;
  hit[2] = p0[2] + u[2] * sI;
  return true;
}

// Box of the part of triangle v on each side of the plane, clamped to the
// triangle's box [lo, hi]: the side's own vertices in order, then the
// plane's hits in (left vertex, right vertex) order, shared by both sides.
struct ClipBox {
  float lo[2][3], hi[2][3];
  bool any[2];
  __device__ __forceinline__ void add(int s, const float* p) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      lo[s][d] = any[s] ? ref_min(lo[s][d], p[d]) : p[d];
      hi[s][d] = any[s] ? ref_max(hi[s][d], p[d]) : p[d];
    }
    any[s] = true;
  }
};
__device__ __forceinline__ void clip_boxes(const float v[3][3], const float lo[3], const float hi[3], int axis,
                                           float split, ClipBox& C) {
  const float pn[3] = {axis == 0 ? 1.f : 0.f, axis == 1 ? 1.f : 0.f, axis == 2 ? 1.f : 0.f};
  const float pp[3] = {pn[0] * split, pn[1] * split, pn[2] * split};
  bool left[3];
  C.any[0] = C.any[1] = false;
#pragma unroll
  for (int s = 0; s < 2; ++s)
#pragma unroll
    for (int d = 0; d < 3; ++d) C.lo[s][d] = C.hi[s][d] = 0.f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    left[k] = pick(v[k], axis) < split;
    if (left[k]) C.add(0, v[k]);
    else C.add(1, v[k]);
  }
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      if (j == k) continue;
      float h[3];
      if (left[j] && !left[k] && edge_plane(v[j], v[k], pp, pn, h)) {
        C.add(0, h);
        C.add(1, h);
      }
    }
#pragma unroll
  for (int s = 0; s < 2; ++s)
    if (C.any[s])
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        C.lo[s][d] = ref_max(C.lo[s][d], lo[d]);
        C.hi[s][d] = ref_min(C.hi[s][d], hi[d]);
      }
}

// Triangles to their children.  sc: exclusive scan of SideOp; a split node's
// children take consecutive ranges, so a left slot is the left count before t
// plus the right count before the node, a right slot the right count before
// t plus the left count up to the node's end.
__global__ void k_part_scatter(TriView V, size_t T, const float* __restrict__ g, const float* __restrict__ kiso,
                               const uint32_t* __restrict__ tb, const Decision* __restrict__ dec,
                               const uint64_t* __restrict__ nsc, const uint64_t* __restrict__ sc, float* lo2,
                               float* hi2, uint32_t* tri2, uint32_t* node2, size_t cap2) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T) return;
  const uint32_t n = V.node[t];
  const Decision d = dec[n];
  if (d.axis < 0) return;
  float blo[3], bhi[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    blo[a] = V.lo[a * V.cap + t];
    bhi[a] = V.hi[a * V.cap + t];
  }
  const float mn = pick(blo, d.axis), mx = pick(bhi, d.axis);
  bool go[2];
  sides_of(mn, mx, d, &go[0], &go[1]);
  if (!go[0] && !go[1]) return;
  const uint32_t tri = V.tri[t];
  const uint64_t s = sc[t];
  const size_t pos[2] = {(size_t)lo32(s) + hi32(sc[tb[n]]), (size_t)hi32(s) + lo32(sc[tb[n + 1]])};
  const uint32_t child = 2 * lo32(nsc[n]);
  ClipBox C;
  if (mn < d.split && mx > d.split) {
    float v[3][3];
    proxy_triangle(g, kiso, tri, v);
    clip_boxes(v, blo, bhi, d.axis, d.split, C);
  } else {
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        C.lo[k][a] = blo[a];
        C.hi[k][a] = bhi[a];
      }
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    if (!go[k]) continue;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo2[a * cap2 + pos[k]] = C.lo[k][a];
      hi2[a * cap2 + pos[k]] = C.hi[k][a];
    }
    tri2[pos[k]] = tri;
    node2[pos[k]] = child + k;
  }
}

// A node of the finished level, as the numbering reads it.
struct Rec {
  int axis;        // -1: leaf
  uint32_t split;  // split bits
  uint32_t child;  // index of the left child in the next level
  uint32_t leaf_off, leaf_cnt;
};

// Per node: its record, and for split nodes the children's boxes and first
// triangles.
__global__ void k_children(const uint32_t* __restrict__ tb, const uint32_t* __restrict__ rb, uint32_t N,
                           const Decision* __restrict__ dec, const uint64_t* __restrict__ nsc,
                           const uint64_t* __restrict__ sc, uint32_t pool_base, const float* __restrict__ nlo,
                           const float* __restrict__ nhi, float* clo, float* chi, uint32_t* ctb, Rec* rec,
                           LevelSum* sum) {
  const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t ids = 0;
  if (n < N) {
    const Decision d = dec[n];
    const uint64_t e = nsc[n];
    const uint32_t G = rb[n + 1] - rb[n];
    Rec r;
    r.axis = d.axis;
    r.split = __float_as_uint(d.split);
    r.child = 2 * lo32(e);
    r.leaf_off = pool_base + hi32(e);
    r.leaf_cnt = d.axis < 0 ? G : 0u;
    rec[n] = r;
    if (d.axis >= 0) {
      ids = G;
      const uint64_t s0 = sc[tb[n]], s1 = sc[tb[n + 1]];
      ctb[r.child] = lo32(s0) + hi32(s0);
      ctb[r.child + 1] = lo32(s1) + hi32(s0);
#pragma unroll
      for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const float l = nlo[3ull * n + k], h = nhi[3ull * n + k];
          clo[3ull * (r.child + s) + k] = s == 1 && k == d.axis ? d.split : l;
          chi[3ull * (r.child + s) + k] = s == 0 && k == d.axis ? d.split : h;
        }
    }
    if (n == N - 1) {
      const uint64_t ne = nsc[N], se = sc[tb[N]];
      sum->triangles = (unsigned long long)lo32(se) + hi32(se);
      sum->n_split = lo32(ne);
      sum->leaf_ids = hi32(ne);
      ctb[2 * lo32(ne)] = lo32(se) + hi32(se);
    }
  }
  ids = __reduce_max_sync(0xFFFFFFFFu, ids);
  if ((threadIdx.x & 31) == 0 && ids) atomicMax(&sum->max_ids, ids);
}

__global__ void k_leaf_ids(const uint32_t* __restrict__ run_start, const uint32_t* __restrict__ run_node,
                           const uint32_t* __restrict__ tri, const uint32_t* __restrict__ ids,
                           const uint32_t* __restrict__ is_split, const uint32_t* __restrict__ rb, uint32_t N,
                           const uint64_t* __restrict__ nsc, uint32_t* pool) {
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < rb[N]; r += gridDim.x * blockDim.x) {
    const uint32_t n = run_node[r];
    if (is_split[n]) continue;
    pool[hi32(nsc[n]) + (r - rb[n])] = ids[tri[run_start[r]] / kFaces];
  }
}

// ------------------------------------------------------------ numbering
// Bottom up: inner nodes and leaf IDs of every subtree.
__global__ void k_subtree(const Rec* __restrict__ rec, uint32_t N, const uint2* __restrict__ below, uint2* own,
                          uint32_t* max_leaf) {
  const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t leaf = 0;
  if (n < N) {
    const Rec r = rec[n];
    if (r.axis < 0) {
      own[n] = make_uint2(0u, r.leaf_cnt);
      leaf = r.leaf_cnt;
    } else {
      const uint2 a = below[r.child], b = below[r.child + 1];
      own[n] = make_uint2(1u + a.x + b.x, a.y + b.y);
    }
  }
  leaf = __reduce_max_sync(0xFFFFFFFFu, leaf);
  if ((threadIdx.x & 31) == 0 && leaf) atomicMax(max_leaf, leaf);
}

// Where a node goes: its slot, the number of inner nodes before it and of
// leaf IDs before it in depth-first, left-first order.
struct Place {
  uint32_t slot, rank, ids;
};
// Top down: the reference allocates a child pair when it pops the parent, so
// the pair of the inner node of rank k is (1 + 2k, 2 + 2k).
__global__ void k_place(const Rec* __restrict__ rec, uint32_t N, const uint2* __restrict__ below,
                        const Place* __restrict__ at, Place* next, uint2* nodes, const uint32_t* __restrict__ pool,
                        uint32_t* offsets) {
  const uint32_t n = (blockIdx.x * blockDim.x + threadIdx.x) >> 3;  // 8 lanes per node copy a leaf's IDs
  const uint32_t lane = threadIdx.x & 7u;
  if (n >= N) return;
  const Rec r = rec[n];
  const Place p = at[n];
  if (r.axis < 0) {
    if (lane == 0) nodes[p.slot] = make_uint2((r.leaf_cnt << 3) | 3u, p.ids);
    for (uint32_t i = lane; i < r.leaf_cnt; i += 8) offsets[p.ids + i] = pool[r.leaf_off + i];
  } else if (lane == 0) {
    const uint32_t c = 1u + 2u * p.rank;
    const uint2 l = below[r.child];
    nodes[p.slot] = make_uint2((c << 3) | (uint32_t)r.axis, r.split);
    next[r.child] = Place{c, p.rank + 1u, p.ids};
    next[r.child + 1] = Place{c + 1u, p.rank + 1u + l.x, p.ids + l.y};
  }
}

template <int NT, int CAP>
void launch_search_block(Stream& S, const Params& P, const uint32_t* list, const uint32_t* count, uint32_t most,
                         const uint32_t* tb, const uint32_t* rb, const uint32_t* ridx, const TriView& V,
                         const float* nlo, const float* nhi, Decision* dec, uint32_t* is_split) {
  const int bytes = (int)sizeof(SearchMem<NT, CAP>);
  S.check(cudaFuncSetAttribute(k_search_block<NT, CAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  const unsigned grid = std::max(1u, std::min(most, 4096u));
  k_search_block<NT, CAP><<<grid, NT, bytes, S.s>>>(P, list, count, tb, rb, ridx, V, nlo, nhi, dec, is_split);
}

// Host threads of the steps around the build.  Reading 500k records for their
// proxies took 6.0 ms on one thread and 1 ms on eight; the first touch of the
// result's pages by the copy engine 2.4 ms for 40 MB against 0.8.
constexpr uint32_t kHostThreads = 8;
template <typename F>
void host_parallel(uint32_t n, F fn) {
  std::vector<std::thread> t;
  uint32_t r = 1;
  try {
    t.reserve(n);
    for (; r < n; ++r) t.emplace_back(fn, r);
  } catch (const std::system_error&) {  // no more threads: the rest runs here
  } catch (const std::bad_alloc&) {     // nor memory for one
  }
  fn(0u);
  for (uint32_t k = r; k < n; ++k) fn(k);
  for (auto& x : t) x.join();
}

// malloc with the pages of a large array touched by several threads.
void* host_array(size_t bytes) {
  char* p = static_cast<char*>(malloc(bytes));
  if (!p || bytes < (4u << 20)) return p;
  const long page = std::max(4096l, sysconf(_SC_PAGESIZE));
  host_parallel(kHostThreads, [=](uint32_t r) {
    const size_t lo = bytes / kHostThreads * r, hi = r + 1 == kHostThreads ? bytes : bytes / kHostThreads * (r + 1);
    for (size_t i = lo; i < hi; i += (size_t)page) reinterpret_cast<volatile char*>(p)[i] = 0;
  });
  return p;
}

}  // namespace

int build_tree_gpu(const float* gauss, uint32_t n, const BuildParams& bp, kdgr_tree* out, BuildStats* stats,
                   std::string& err) {
  using clk = std::chrono::steady_clock;
  auto t0 = clk::now();
  // the host arrays of the result: released on every exit but the last
  struct HostArrays {
    void *nodes = nullptr, *offsets = nullptr, *valid = nullptr;
    ~HostArrays() {
      free(nodes);
      free(offsets);
      free(valid);
    }
  } H;
  H.valid = calloc((size_t)n + 1, 1);
  if (!H.valid) throw std::bad_alloc();
  uint8_t* valid = static_cast<uint8_t*>(H.valid);
  // per-Gaussian proxy scale on the host (the host builder's function), in
  // ranges: the scales first, then each range's fields after those before it
  std::vector<float> kall(n);
  const uint32_t n_ranges = std::max(1u, std::min(kHostThreads, n / 16384u));
  std::vector<uint32_t> first(n_ranges + 1, 0u);
  auto range_lo = [&](uint32_t r) { return (uint32_t)((uint64_t)n * r / n_ranges); };
  host_parallel(n_ranges, [&](uint32_t r) {
    uint32_t c = 0;
    for (uint32_t i = range_lo(r); i < range_lo(r + 1); ++i) {
      valid[i] = proxy_kiso(gauss + (size_t)i * 64, &kall[i]) ? 1 : 0;
      c += valid[i];
    }
    first[r + 1] = c;
  });
  for (uint32_t r = 0; r < n_ranges; ++r) first[r + 1] += first[r];
  const uint32_t n_valid = first[n_ranges];
  std::vector<float> gv((size_t)n_valid * 10), kiso(n_valid);
  std::vector<uint32_t> ids(n_valid);
  host_parallel(n_ranges, [&](uint32_t r) {
    size_t j = first[r];
    for (uint32_t i = range_lo(r); i < range_lo(r + 1); ++i) {
      if (!valid[i]) continue;
      const float* g = gauss + (size_t)i * 64;
      const float f[10] = {g[0], g[1], g[2], g[4], g[5], g[6], g[8], g[9], g[10], g[11]};
      memcpy(&gv[10 * j], f, sizeof f);
      kiso[j] = kall[i];
      ids[j++] = i;
    }
  });
  if (n_valid == 0) {
    err = "every Gaussian is below the opacity cut; nothing to build";
    return KDGR_ERR_INVALID_ARG;
  }
  if ((uint64_t)n_valid * kFaces > 0xFFFFFFF0ull) {
    err = "more than 2^32 proxy triangles";
    return KDGR_ERR_LIMIT;
  }
  bool limit_hit = false;
  Stream S;  // after the host arrays that its copies read and write: it ends before them
  const Params P{bp.max_level,  bp.force_split, bp.isect_cost,
                 bp.sah_mode,   bp.sort_cost,   (bp.isect_cost >= 0.0f && bp.sort_cost >= 0.0f) ? 1 : 0};
  uint32_t depth = 0, n_leaves = 0, max_leaf = 0, n_nodes = 0;
  size_t pool_used = 0;
  float box_lo[3] = {0, 0, 0}, box_hi[3] = {0, 0, 0};
  auto t2 = t0;
  if (S.err == cudaSuccess) {
    S.check(cudaMemcpyToSymbolAsync(c_ico_v, kIcosaVerts, sizeof kIcosaVerts, 0, cudaMemcpyHostToDevice, S.s));
    S.check(cudaMemcpyToSymbolAsync(c_ico_f, kIcosaFaces, sizeof kIcosaFaces, 0, cudaMemcpyHostToDevice, S.s));
    DBuf<float> d_g(S, gv.size()), d_k(S, kiso.size());
    DBuf<uint32_t> d_ids(S, ids.size());
    S.check(cudaMemcpyAsync(d_g.p, gv.data(), gv.size() * 4, cudaMemcpyHostToDevice, S.s));
    S.check(cudaMemcpyAsync(d_k.p, kiso.data(), kiso.size() * 4, cudaMemcpyHostToDevice, S.s));
    S.check(cudaMemcpyAsync(d_ids.p, ids.data(), ids.size() * 4, cudaMemcpyHostToDevice, S.s));
    size_t T = (size_t)n_valid * kFaces;
    TriSet cur;
    cur.alloc(S, T);
    DBuf<uint32_t> d_box(S, 6);
    DBuf<float> nlo(S, 3), nhi(S, 3);
    DBuf<uint32_t> tb(S, 2);
    if (S.err == cudaSuccess) {
      k_proxy<<<grid_for(T, 256), 256, 0, S.s>>>(d_g.p, d_k.p, n_valid, cur.lo.p, cur.hi.p, cur.tri.p, cur.node.p,
                                                 cur.cap);
      const uint32_t box_init[6] = {0xFFFFFFFFu, 0, 0xFFFFFFFFu, 0, 0xFFFFFFFFu, 0};
      S.check(cudaMemcpyAsync(d_box.p, box_init, sizeof box_init, cudaMemcpyHostToDevice, S.s));
      k_scene_box<<<std::min(1024u, grid_for(T, 256)), 256, 0, S.s>>>(view(cur), T, d_box.p);
      k_box_decode<<<1, 32, 0, S.s>>>(d_box.p, nlo.p, nhi.p);
      S.check(cudaMemcpyAsync(box_lo, nlo.p, 12, cudaMemcpyDeviceToHost, S.s));
      S.check(cudaMemcpyAsync(box_hi, nhi.p, 12, cudaMemcpyDeviceToHost, S.s));
      const uint32_t tb0[2] = {0, (uint32_t)T};
      S.check(cudaMemcpyAsync(tb.p, tb0, 8, cudaMemcpyHostToDevice, S.s));
      S.check(cudaGetLastError());
      S.check(cudaStreamSynchronize(S.s));
    }
    auto t1 = clk::now();
    if (stats) stats->proxy_s = std::chrono::duration<double>(t1 - t0).count();
    if (stats) stats->n_triangles = T;
    if (stats) stats->n_valid = n_valid;

    DBuf<uint32_t> pool;
    DBuf<uint8_t> tmp;  // scan and sort workspace
    std::vector<DBuf<Rec>> levels;
    std::vector<uint32_t> level_n;
    uint32_t N = 1, max_ids = n_valid;
    for (int level = 0; N > 0 && S.err == cudaSuccess; ++level) {
#ifdef KDGR_BUILD_TRACE  // compile-time diagnostic: per-level wall time and sizes on stderr
      const auto lt0 = clk::now();
      fprintf(stderr, "[kdbuild_gpu] level %d: %u nodes, %zu triangles, at most %u IDs", level, N, T, max_ids);
#endif
      depth = (uint32_t)level;
      const TriView V = view(cur);
      // 1. runs of (node, ID)
      DBuf<uint32_t> ridx(S, T + 1), run_start(S, T + 1), run_node(S, T + 1), rb(S, (size_t)N + 1), counts(S, kCounts);
      DBuf<LevelSum> d_sum(S, 1);
      if (S.err != cudaSuccess) break;
      exclusive_sum_of(S, tmp, HeadOp{V.tri, V.node, T}, ridx.p, T + 1);
      k_run_scatter<<<grid_for(T, 256), 256, 0, S.s>>>(ridx.p, V.node, T, run_start.p, run_node.p, counts.p, d_sum.p);
      // 2. node classes and split search; large nodes can only appear below a large node
      const bool may_be_big = max_ids > kBlockIds;
      DBuf<Decision> dec(S, N);
      DBuf<uint32_t> is_split(S, (size_t)N + 1), lists(S, 2 * (size_t)N), eG;
      if (may_be_big) eG.alloc(S, (size_t)N + 1);
      if (S.err != cudaSuccess) break;
      const uint32_t warp_ids = N < kFewNodes ? 0u : kWarpIds;
      k_node_setup<<<grid_for((size_t)N + 1, 128), 128, 0, S.s>>>(tb.p, ridx.p, N, level, P.max_level, warp_ids, rb.p,
                                                                  dec.p, is_split.p, lists.p, lists.p + N, counts.p,
                                                                  eG.p);
      if (warp_ids)
        k_search_warp<<<grid_for(N, kSearchWarps), 32 * kSearchWarps, 0, S.s>>>(
            P, N, level, tb.p, rb.p, ridx.p, V, nlo.p, nhi.p, dec.p, is_split.p);
      if (max_ids > std::max(warp_ids, kMinPrim))
        launch_search_block<128, (int)kMidIds>(S, P, lists.p, counts.p + kCntMid, N, tb.p, rb.p, ridx.p, V, nlo.p, nhi.p, dec.p,
                                               is_split.p);
      if (max_ids > kMidIds)
        launch_search_block<512, (int)kBlockIds>(S, P, lists.p + N, counts.p + kCntBlock, N, tb.p, rb.p, ridx.p, V,
                                                 nlo.p, nhi.p, dec.p, is_split.p);
      if (may_be_big) {
        DBuf<uint32_t> grb(S, (size_t)N + 1);
        if (S.err != cudaSuccess) break;
        exclusive_sum(S, tmp, (const uint32_t*)eG.p, grb.p, (size_t)N + 1);
        uint32_t eGT = 0;
        S.check(cudaMemcpyAsync(&eGT, grb.p + N, 4, cudaMemcpyDeviceToHost, S.s));
        S.check(cudaStreamSynchronize(S.s));
        if (eGT > 0) {
          Big B{};
          B.grb = grb.p;
          B.eGn = eG.p;
          B.eG = eGT;
          B.nb = 1;
          while ((1ull << B.nb) < N) ++B.nb;
          DBuf<uint64_t> kmin(S, 3 * (size_t)eGT), kmax(S, 3 * (size_t)eGT), kpl(S, 3 * (size_t)eGT),
              alt(S, 3 * (size_t)eGT);
          DBuf<uint32_t> best32(S, N), hull(S, 6 * (size_t)N);
          DBuf<unsigned long long> best64(S, 2 * (size_t)N);
          DBuf<float2> scores(S, 6 * (size_t)eGT);
          DBuf<Scored> scored(S, kScoredCap);
          if (S.err != cudaSuccess) break;
          uint32_t* const pl_fill = counts.p + kCntPlanar;
          k_run_bounds<<<grid_for(T, 128), 128, 0, S.s>>>(run_start.p, run_node.p, rb.p, N, T, V, B, kmin.p, kmax.p,
                                                          kpl.p, pl_fill);
          S.check(cudaMemcpyAsync(&B.n_pl, pl_fill, 4, cudaMemcpyDeviceToHost, S.s));
          const int end_bit = 32 + B.nb + 2;
          sort_keys(S, tmp, kmin, alt, 3 * (size_t)eGT, end_bit);
          sort_keys(S, tmp, kmax, alt, 3 * (size_t)eGT, end_bit);
          S.check(cudaStreamSynchronize(S.s));
          sort_keys(S, tmp, kpl, alt, B.n_pl, end_bit);
          B.kmin = kmin.p;
          B.kmax = kmax.p;
          B.kpl = kpl.p;
          BigState st{best32.p, best64.p, best64.p + N, hull.p, hull.p + 3 * (size_t)N, scored.p, counts.p + kCntScored};
          const unsigned ge = grid_for(6 * (size_t)eGT, 256), gt = grid_for(T, 256), gn = grid_for(N, 128);
          k_big_init<<<gn, 128, 0, S.s>>>(P, B, tb.p, N, st);
          k_event_scores<<<ge, 256, 0, S.s>>>(P, B, tb.p, nlo.p, nhi.p, scores.p, st);
          k_event_exact<true><<<ge, 256, 0, S.s>>>(P, B, tb.p, nlo.p, nhi.p, scores.p, st);
          k_edge_exact<true><<<gt, 256, 0, S.s>>>(P, B, V, T, tb.p, nlo.p, nhi.p, st);
          k_scored_first<<<256, 256, 0, S.s>>>(st);
          k_event_exact<false><<<ge, 256, 0, S.s>>>(P, B, tb.p, nlo.p, nhi.p, scores.p, st);
          k_edge_exact<false><<<gt, 256, 0, S.s>>>(P, B, V, T, tb.p, nlo.p, nhi.p, st);
          k_big_choose<<<gn, 128, 0, S.s>>>(B, N, st, dec.p, is_split.p);
        }
      }
      S.check(cudaGetLastError());
      // 3. children: node numbers, leaf ID ranges, triangle ranges
      DBuf<uint64_t> nsc(S, (size_t)N + 1), sc(S, T + 1);
      DBuf<Rec> rec(S, N);
      DBuf<float> clo(S, 6 * (size_t)N), chi(S, 6 * (size_t)N);
      DBuf<uint32_t> ctb(S, 2 * (size_t)N + 1);
      if (S.err != cudaSuccess) break;
      exclusive_sum_of(S, tmp, NodeOp{is_split.p, rb.p, N}, nsc.p, (size_t)N + 1);
      exclusive_sum_of(S, tmp, SideOp{V, dec.p, T}, sc.p, T + 1);
      k_children<<<grid_for(N, 128), 128, 0, S.s>>>(tb.p, rb.p, N, dec.p, nsc.p, sc.p, (uint32_t)pool_used, nlo.p,
                                                    nhi.p, clo.p, chi.p, ctb.p, rec.p, d_sum.p);
      LevelSum sum{};
      S.check(cudaMemcpyAsync(&sum, d_sum.p, sizeof sum, cudaMemcpyDeviceToHost, S.s));
      S.check(cudaStreamSynchronize(S.s));
      if (S.err != cudaSuccess) break;
      // 4. leaves: their run IDs into the pool
      if (pool_used + sum.leaf_ids > pool.n) {
        DBuf<uint32_t> bigger(S, std::max(pool.n * 2, pool_used + sum.leaf_ids + 1024));
        if (pool_used && S.err == cudaSuccess)
          S.check(cudaMemcpyAsync(bigger.p, pool.p, pool_used * 4, cudaMemcpyDeviceToDevice, S.s));
        pool = std::move(bigger);
        if (S.err != cudaSuccess) break;
      }
      if (sum.leaf_ids)
        k_leaf_ids<<<std::min(grid_for(T, 256), 4096u), 256, 0, S.s>>>(run_start.p, run_node.p, V.tri, d_ids.p,
                                                                       is_split.p, rb.p, N, nsc.p, pool.p + pool_used);
      pool_used += sum.leaf_ids;
      levels.push_back(std::move(rec));
      level_n.push_back(N);
      // 5. partition into the next level
      if (sum.n_split > 0) {
        if (sum.triangles > 0xFFFFFFF0ull || pool_used > 0xFFFFFFF0ull) {
          err = "more than 2^32 triangle references in one level";
          limit_hit = true;
          break;
        }
        TriSet nxt;
        nxt.alloc(S, std::max<size_t>(sum.triangles, 1));
        if (S.err != cudaSuccess) break;
        k_part_scatter<<<grid_for(T, 256), 256, 0, S.s>>>(V, T, d_g.p, d_k.p, tb.p, dec.p, nsc.p, sc.p, nxt.lo.p,
                                                          nxt.hi.p, nxt.tri.p, nxt.node.p, nxt.cap);
        S.check(cudaGetLastError());
        cur = std::move(nxt);
        nlo = std::move(clo);
        nhi = std::move(chi);
        tb = std::move(ctb);
      }
      N = 2 * sum.n_split;
      T = sum.triangles;
      max_ids = sum.max_ids;
#ifdef KDGR_BUILD_TRACE
      cudaStreamSynchronize(S.s);
      fprintf(stderr, ", %.2f ms\n", std::chrono::duration<double, std::milli>(clk::now() - lt0).count());
#endif
    }
    // number as the reference allocates: child pairs in depth-first,
    // left-first order; leaf ID lists in the same order
    if (S.err == cudaSuccess && !limit_hit) {
      const int L = (int)levels.size();
      std::vector<DBuf<uint2>> sub(L);
      DBuf<uint32_t> d_max(S, 1);
      d_max.zero();
      for (int l = L - 1; l >= 0 && S.err == cudaSuccess; --l) {
        sub[l].alloc(S, level_n[l]);
        if (S.err != cudaSuccess) break;
        k_subtree<<<grid_for(level_n[l], 128), 128, 0, S.s>>>(levels[l].p, level_n[l],
                                                              l + 1 < L ? sub[l + 1].p : nullptr, sub[l].p, d_max.p);
      }
      uint2 total = make_uint2(0u, 0u);
      if (S.err == cudaSuccess) {
        S.check(cudaMemcpyAsync(&total, sub[0].p, sizeof total, cudaMemcpyDeviceToHost, S.s));
        S.check(cudaMemcpyAsync(&max_leaf, d_max.p, 4, cudaMemcpyDeviceToHost, S.s));
        S.check(cudaStreamSynchronize(S.s));
      }
      t2 = clk::now();
      if (S.err == cudaSuccess) {
        n_leaves = total.x + 1u;
        n_nodes = 1u + 2u * total.x;
        DBuf<uint2> d_nodes(S, n_nodes);
        DBuf<uint32_t> d_off(S, pool_used + 1);
        DBuf<Place> at(S, 1), next;
        at.zero();  // the root: slot 0, no inner node and no ID before it
        for (int l = 0; l < L && S.err == cudaSuccess; ++l) {
          next.alloc(S, l + 1 < L ? level_n[l + 1] : 1);
          if (S.err != cudaSuccess) break;
          k_place<<<grid_for(8ull * level_n[l], 256), 256, 0, S.s>>>(levels[l].p, level_n[l],
                                                                     l + 1 < L ? sub[l + 1].p : nullptr, at.p, next.p,
                                                                     d_nodes.p, pool.p, d_off.p);
          at = std::move(next);
        }
        S.check(cudaGetLastError());
        H.nodes = host_array(8ull * n_nodes + 4);
        H.offsets = host_array(4 * pool_used + 4);
        if (H.nodes && H.offsets && S.err == cudaSuccess) {
          S.check(cudaMemcpyAsync(H.nodes, d_nodes.p, 8ull * n_nodes, cudaMemcpyDeviceToHost, S.s));
          if (pool_used)
            S.check(cudaMemcpyAsync(H.offsets, d_off.p, 4 * pool_used, cudaMemcpyDeviceToHost, S.s));
        }
      }
    }
    S.check(cudaStreamSynchronize(S.s));
  }  // device buffers are returned to the pool here
  const cudaError_t e = S.err;
  if (limit_hit && e == cudaSuccess) return KDGR_ERR_LIMIT;
  if (e != cudaSuccess) {
    cudaGetLastError();
    if (err.empty()) err = std::string("CUDA error in the device build: ") + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? KDGR_ERR_OUT_OF_MEMORY : KDGR_ERR_CUDA;
  }
  if (!H.nodes || !H.offsets) throw std::bad_alloc();
  memset(out, 0, sizeof(*out));
  out->nodes = static_cast<uint32_t*>(H.nodes);
  out->offsets = static_cast<uint32_t*>(H.offsets);
  out->valid = valid;
  H.nodes = H.offsets = H.valid = nullptr;
  out->n_nodes = n_nodes;
  out->n_offsets = (uint32_t)pool_used;
  for (int a = 0; a < 3; ++a) {
    out->aabb[a] = box_lo[a];
    out->aabb[3 + a] = box_hi[a];
  }
  out->depth = depth;
  out->n_leaves = n_leaves;
  out->max_leaf = max_leaf;
  out->n_gaussians = n;
  auto t3 = clk::now();
  if (stats) {
    stats->build_s = std::chrono::duration<double>(t2 - t0).count() - stats->proxy_s;
    stats->serialize_s = std::chrono::duration<double>(t3 - t2).count();
  }
  return KDGR_OK;
}

}  // namespace kdgr
