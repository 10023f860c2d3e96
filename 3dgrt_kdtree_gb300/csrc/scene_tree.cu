// scene_tree.cu -- the tree side of a scene upload, on the device.
//
// The caller's tree (host arrays, the reference's layout) is copied as it is
// and checked, relaid out and expanded into leaf-order ID lists by kernels:
//   * breadth first from the root, one level per launch: child and leaf
//     ranges, axis fields and nodes reached twice (one bit per node) are
//     checked, and the reached nodes are listed level by level.  Any fault
//     only raises a flag; the host check of the same tree then names it;
//   * the fast forms' node order (top kTopLevels levels breadth first, the
//     rest depth first by subtree, children adjacent) follows from subtree
//     sums taken bottom up and pair numbers handed down;
//   * leaf word y of the relaid tree and the padded ID lists follow from one
//     scan over the relaid nodes; the packed form's two streams from another.
//
// What bounds it: nothing but latency -- a 100 MB tree is read a few times
// from HBM -- so the steps are few launches with two read-backs, not fused
// further.  Opening a scene (upload of the plain and fast forms and a 256x256
// frame, GB300): 200k Gaussians 11.3 -> 1.8 ms against the serial host passes
// it replaces; the 1M scene's upload 80 -> 2.5 ms, its packed form 227 -> 3.0.
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "kdgr_internal.h"
#include "scene.h"

namespace kdgr {
namespace {

constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr int kTopLevels = 10;  // 2047 nodes at most in the breadth-first top

// Counters of one upload.
struct TreeState {
  uint32_t tail;      // nodes listed
  uint32_t bad;       // some check failed
  uint32_t max_leaf, n_leaves;  // over all nodes given
  uint32_t blocks;    // blocks of the running level that are done
};

// One node's checks; returns its left child, or kNone for a leaf or a fault.
__device__ __forceinline__ uint32_t checked_child(uint2 nd, uint32_t n_nodes, uint32_t n_offsets, uint32_t* seen,
                                                  TreeState* st) {
  if ((nd.x & 7u) == 3u) {
    if ((uint64_t)nd.y + (nd.x >> 3) > n_offsets) st->bad = 1u;
    return kNone;
  }
  const uint32_t c = nd.x >> 3;
  if ((nd.x & 4u) != 0u || (nd.x & 3u) == 3u || c == 0u || (uint64_t)c + 1 >= n_nodes) {
    st->bad = 1u;
    return kNone;
  }
  const uint32_t a = atomicOr(&seen[c >> 5], 1u << (c & 31u)) & (1u << (c & 31u));
  const uint32_t b = atomicOr(&seen[(c + 1) >> 5], 1u << ((c + 1) & 31u)) & (1u << ((c + 1) & 31u));
  if (a | b) {
    st->bad = 1u;
    return kNone;
  }
  return c;
}

// Levels 0 .. kTopLevels in breadth-first order, by one block.  list: the
// nodes reached; cpos: list position of a node's left child (kNone: leaf);
// ls[d]: list position of level d's first node.
__global__ void __launch_bounds__(1024) k_top(const uint2* __restrict__ nodes, uint32_t n_nodes, uint32_t n_offsets,
                                              uint32_t* seen, uint32_t* list, uint32_t* cpos, uint32_t* ls,
                                              TreeState* st) {
  using Scan = cub::BlockScan<uint32_t, 1024>;
  __shared__ typename Scan::TempStorage tmp;
  const uint32_t i = threadIdx.x;
  if (i == 0) {
    list[0] = 0u;
    atomicOr(&seen[0], 1u);
  }
  __syncthreads();
  uint32_t s = 0, e = 1;
  for (int d = 0; d < kTopLevels; ++d) {
    uint32_t c = kNone;
    if (s + i < e) c = checked_child(nodes[list[s + i]], n_nodes, n_offsets, seen, st);
    uint32_t rank, total;
    Scan(tmp).ExclusiveSum(c != kNone ? 1u : 0u, rank, total);
    if (s + i < e) {
      cpos[s + i] = c != kNone ? e + 2 * rank : kNone;
      if (c != kNone) {
        list[e + 2 * rank] = c;
        list[e + 2 * rank + 1] = c + 1;
      }
    }
    if (i == 0) ls[d] = s;
    s = e;
    e += 2 * total;
    __syncthreads();
  }
  if (i == 0) {
    ls[kTopLevels] = s;
    ls[kTopLevels + 1] = e;
    st->tail = e;
  }
}

// Level l >= kTopLevels: its nodes' children are appended (in any order: node
// numbers come from the tree, not from list positions); the last block done
// closes the next level.
__global__ void k_expand(const uint2* __restrict__ nodes, uint32_t n_nodes, uint32_t n_offsets, uint32_t* seen,
                         uint32_t* list, uint32_t* cpos, uint32_t* ls, int l, TreeState* st) {
  const uint32_t s = ls[l], e = ls[l + 1];
  const unsigned lane = threadIdx.x & 31u;
  for (uint32_t b = s + blockIdx.x * blockDim.x; b < e; b += gridDim.x * blockDim.x) {
    const uint32_t i = b + threadIdx.x;
    uint32_t c = kNone;
    if (i < e) c = checked_child(nodes[list[i]], n_nodes, n_offsets, seen, st);
    const unsigned m = __ballot_sync(0xFFFFFFFFu, c != kNone);
    uint32_t at = 0;
    if (m && lane == 0) at = atomicAdd(&st->tail, 2u * __popc(m));
    at = __shfl_sync(0xFFFFFFFFu, at, 0) + 2u * __popc(m & ((1u << lane) - 1u));
    if (i < e) cpos[i] = c != kNone ? at : kNone;
    if (c != kNone) {
      list[at] = c;
      list[at + 1] = c + 1;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&st->blocks, 1u) == gridDim.x - 1) {
      st->blocks = 0u;
      ls[l + 2] = atomicAdd(&st->tail, 0u);
    }
  }
}

__global__ void k_leaf_stats(const uint2* __restrict__ nodes, uint32_t n, TreeState* st) {
  uint32_t leaves = 0, most = 0;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t x = nodes[i].x;
    if ((x & 7u) == 3u) {
      ++leaves;
      most = max(most, x >> 3);
    }
  }
  leaves = __reduce_add_sync(0xFFFFFFFFu, leaves);
  most = __reduce_max_sync(0xFFFFFFFFu, most);
  if ((threadIdx.x & 31) == 0 && leaves) {
    atomicAdd(&st->n_leaves, leaves);
    atomicMax(&st->max_leaf, most);
  }
}

// Lanes that share one leaf's ID list.
constexpr uint32_t kLeafLanes = 8;

// Every ID of every reached leaf is below n_gauss (leaf ranges have been
// checked; a fault leaves the flag set and the ranges are not read).
__global__ void k_check_ids(const uint2* __restrict__ nodes, const uint32_t* __restrict__ list,
                            const uint32_t* __restrict__ offsets, uint32_t n_gauss, TreeState* st) {
  if (st->bad) return;
  const uint32_t n = st->tail, lane = threadIdx.x % kLeafLanes;
  bool bad = false;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / kLeafLanes; i < n;
       i += gridDim.x * blockDim.x / kLeafLanes) {
    const uint2 nd = nodes[list[i]];
    if ((nd.x & 7u) != 3u) continue;
    for (uint32_t k = lane; k < (nd.x >> 3); k += kLeafLanes) bad |= offsets[nd.y + k] >= n_gauss;
  }
  if (bad) st->bad = 1u;
}

// Bottom up: inner nodes of every subtree.
__global__ void k_sums(const uint32_t* __restrict__ cpos, const uint32_t* __restrict__ ls, int l, uint32_t* sub) {
  for (uint32_t i = ls[l] + blockIdx.x * blockDim.x + threadIdx.x; i < ls[l + 1]; i += gridDim.x * blockDim.x) {
    const uint32_t c = cpos[i];
    sub[i] = c == kNone ? 0u : 1u + sub[c] + sub[c + 1];
  }
}

// New numbers of the top (its list positions) and of the child pairs of
// level kTopLevels: one depth-first run of pairs per subtree, in order.
__global__ void __launch_bounds__(1024) k_place_top(const uint32_t* __restrict__ cpos, const uint32_t* __restrict__ ls,
                                                    const uint32_t* __restrict__ sub, uint32_t* idx, uint32_t* pair) {
  using Scan = cub::BlockScan<uint32_t, 1024>;
  __shared__ typename Scan::TempStorage tmp;
  const uint32_t i = threadIdx.x, s = ls[kTopLevels], e = ls[kTopLevels + 1];
  for (uint32_t k = i; k < e; k += 1024) {
    idx[k] = k;
    if (k < s) pair[k] = cpos[k];
  }
  uint32_t before;
  const uint32_t own = s + i < e && cpos[s + i] != kNone ? sub[s + i] : 0u;
  Scan(tmp).ExclusiveSum(own, before);
  if (s + i < e) pair[s + i] = e + 2 * before;
}

// Top down: a node's children take its pair, the left subtree's pairs
// follow, then the right's.
__global__ void k_place(const uint32_t* __restrict__ cpos, const uint32_t* __restrict__ ls,
                        const uint32_t* __restrict__ sub, int l, uint32_t* idx, uint32_t* pair) {
  for (uint32_t i = ls[l] + blockIdx.x * blockDim.x + threadIdx.x; i < ls[l + 1]; i += gridDim.x * blockDim.x) {
    const uint32_t c = cpos[i];
    if (c == kNone) continue;
    const uint32_t p = pair[i];
    idx[c] = p;
    idx[c + 1] = p + 1;
    pair[c] = p + 2;
    pair[c + 1] = p + 2 + 2 * sub[c];
  }
}

__global__ void k_relaid(const uint2* __restrict__ nodes, const uint32_t* __restrict__ list, uint32_t n,
                         const uint32_t* __restrict__ cpos, const uint32_t* __restrict__ idx,
                         const uint32_t* __restrict__ pair, uint2* out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint2 nd = nodes[list[i]];
  if (cpos[i] != kNone) nd.x = (pair[i] << 3) | (nd.x & 3u);
  out[idx[i]] = nd;
}

struct PairOp {  // pairs of a relaid node's leaf
  const uint2* nodes;
  uint64_t n;
  __device__ uint64_t operator()(uint64_t i) const {
    if (i >= n) return 0ull;
    const uint32_t x = nodes[i].x;
    return (x & 7u) == 3u ? ((x >> 3) + 1u) >> 1 : 0u;
  }
};

// Padded leaf-order IDs; leaf word y becomes the leaf's first pair.
__global__ void k_leaf_gids(uint2* nodes, uint32_t n, const uint64_t* __restrict__ first,
                            const uint32_t* __restrict__ offsets, uint32_t* gid) {
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / kLeafLanes, lane = threadIdx.x % kLeafLanes;
  uint2 nd = make_uint2(0u, 0u);
  if (i < n) nd = nodes[i];
  __syncwarp();  // every lane of the leaf has read its offset
  if (i >= n || (nd.x & 7u) != 3u) return;
  const uint64_t p = first[i];
  const uint32_t cnt = nd.x >> 3;
  for (uint32_t k = lane; k < cnt + (cnt & 1u); k += kLeafLanes)
    gid[2 * p + k] = k < cnt ? offsets[nd.y + k] : kPadGid;
  if (lane == 0) nodes[i].y = (uint32_t)p;
}

// First pair of every leaf under its number in the tree as given.
__global__ void k_leaf_first(const uint32_t* __restrict__ list, const uint32_t* __restrict__ cpos,
                             const uint32_t* __restrict__ idx, uint32_t n, const uint64_t* __restrict__ first,
                             uint32_t* out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && cpos[i] == kNone) out[list[i]] = (uint32_t)first[idx[i]];
}

struct FlagOp {
  const uint8_t* flag;
  uint64_t n;
  __device__ uint32_t operator()(uint64_t i) const { return i < n && flag[i] ? 1u : 0u; }
};
__global__ void k_aniso_index(const uint8_t* __restrict__ flag, uint32_t n, uint32_t* aidx) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && !flag[i]) aidx[i] = kNone;
}

// Packed form: plain entries (low word) and flagged entries (high word) of
// every relaid leaf, as pairs.
__global__ void k_split_counts(const uint2* __restrict__ nodes, uint32_t n, const uint32_t* __restrict__ gid,
                               const uint8_t* __restrict__ flag, uint64_t* cnt) {
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / kLeafLanes, lane = threadIdx.x % kLeafLanes;
  uint2 nd = make_uint2(0u, 0u);
  if (i < n) nd = nodes[i];
  const bool leaf = (nd.x & 7u) == 3u;
  uint32_t f = 0;
  if (leaf)
    for (uint32_t k = lane; k < (nd.x >> 3); k += kLeafLanes) f += flag[gid[2ull * nd.y + k]] ? 1u : 0u;
  for (uint32_t o = 1; o < kLeafLanes; o <<= 1) f += __shfl_xor_sync(0xFFFFFFFFu, f, o);
  if (i > n || lane != 0) return;
  cnt[i] = leaf ? (uint64_t)(((nd.x >> 3) - f + 1u) >> 1) | (uint64_t)((f + 1u) >> 1) << 32 : 0ull;  // cnt[n] = 0
}

// The two streams of every leaf, entries in leaf order, each padded to whole
// pairs; the packed tree's leaf words and the per-node aux words.
__global__ void k_split_fill(const uint2* __restrict__ nodes, uint32_t n, const uint32_t* __restrict__ gid,
                             const uint8_t* __restrict__ flag, const uint64_t* __restrict__ first, uint2* nodes_p,
                             uint2* aux, uint32_t* gid_plain, uint32_t* gid_flag) {
  const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / kLeafLanes, lane = threadIdx.x % kLeafLanes;
  uint2 nd = make_uint2(0u, 0u);
  if (i < n) nd = nodes[i];
  const bool leaf = (nd.x & 7u) == 3u;
  const uint32_t cnt = leaf ? nd.x >> 3 : 0u;
  const uint64_t at = i < n ? first[i] : 0ull;
  const uint64_t pp = (uint32_t)at, fp = at >> 32;
  uint32_t np = 0, nf = 0;
  const unsigned shift = (threadIdx.x & 31u) & ~(kLeafLanes - 1u), below = (1u << lane) - 1u;
  const uint32_t rounds = __reduce_max_sync(0xFFFFFFFFu, (cnt + kLeafLanes - 1) / kLeafLanes);
  for (uint32_t r = 0; r < rounds; ++r) {
    const uint32_t k = r * kLeafLanes + lane;
    const uint32_t g = k < cnt ? gid[2ull * nd.y + k] : 0u;
    const bool f = k < cnt && flag[g], p = k < cnt && !flag[g];
    const unsigned mf = (__ballot_sync(0xFFFFFFFFu, f) >> shift) & ((1u << kLeafLanes) - 1u);
    const unsigned mp = (__ballot_sync(0xFFFFFFFFu, p) >> shift) & ((1u << kLeafLanes) - 1u);
    if (p) gid_plain[2 * pp + np + __popc(mp & below)] = g;
    if (f) gid_flag[2 * fp + nf + __popc(mf & below)] = g;
    np += __popc(mp);
    nf += __popc(mf);
  }
  if (i >= n || lane != 0) return;
  if (leaf) {
    if (np & 1u) gid_plain[2 * pp + np] = kPadGid;
    if (nf & 1u) gid_flag[2 * fp + nf] = kPadGid;
    nodes_p[i] = make_uint2((np << 3) | 3u, (uint32_t)pp);
    aux[i] = make_uint2((uint32_t)fp, nf);
  } else {
    nodes_p[i] = nd;
    aux[i] = make_uint2(0u, 0u);
  }
}

constexpr unsigned kSweep = 152 * 4;  // blocks of the kernels whose range only the device knows
unsigned blocks_for(uint64_t n, unsigned per) { return (unsigned)std::max<uint64_t>(1, (n + per - 1) / per); }

template <typename It, typename T>
cudaError_t scan_to(WorkMem& W, It in, T* out, uint64_t n) {
  size_t bytes = 0;
  cudaError_t e = cub::DeviceScan::ExclusiveSum(nullptr, bytes, in, out, (int64_t)n, W.st);
  void* tmp = nullptr;
  if (e == cudaSuccess) tmp = W.take<uint8_t>(bytes);
  if (e == cudaSuccess) e = W.err;
  if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(tmp, bytes, in, out, (int64_t)n, W.st);
  return e;
}
template <typename Op, typename T>
cudaError_t scan_of(WorkMem& W, Op op, T* out, uint64_t n) {
  return scan_to(W, thrust::make_transform_iterator(thrust::counting_iterator<uint64_t>(0), op), out, n);
}

}  // namespace

cudaError_t tree_check(WorkMem& W, const uint2* d_nodes, uint32_t n_nodes, const uint32_t* d_offsets,
                       uint32_t n_offsets, uint32_t n_gauss, TreeLists& L) {
  const size_t n = n_nodes;
  L.list = W.take<uint32_t>(n);
  L.cpos = W.take<uint32_t>(n);
  L.ls = W.take<uint32_t>(n + kTopLevels + 40);  // a level holds at least two nodes, the root apart
  uint32_t* seen = W.take<uint32_t>(n / 32 + 2);
  TreeState* st = W.take<TreeState>(1);
  cudaError_t e = W.err;
  if (e == cudaSuccess) e = cudaMemsetAsync(seen, 0, (n / 32 + 2) * 4, W.st);
  if (e == cudaSuccess) e = cudaMemsetAsync(st, 0, sizeof(TreeState), W.st);
  if (e != cudaSuccess) return e;
  k_leaf_stats<<<std::min(kSweep, blocks_for(n, 256)), 256, 0, W.st>>>(d_nodes, n_nodes, st);
  k_top<<<1, 1024, 0, W.st>>>(d_nodes, n_nodes, n_offsets, seen, L.list, L.cpos, L.ls, st);
  // level by level, a few levels per read-back: the builders' trees end
  // within the first (at most 24 levels by default)
  int l = kTopLevels;
  uint32_t edge[2] = {0, 0};
  TreeState h{};
  const unsigned grid = std::min(kSweep, blocks_for(n, 256));
  do {
    const int stop = l + (l == kTopLevels ? 15 : 32);
    for (; l < stop && (size_t)l + 2 < n + kTopLevels + 40; ++l)
      k_expand<<<grid, 256, 0, W.st>>>(d_nodes, n_nodes, n_offsets, seen, L.list, L.cpos, L.ls, l, st);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(edge, L.ls + l, 8, cudaMemcpyDeviceToHost, W.st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(W.st);
    if (e != cudaSuccess) return e;
  } while (edge[0] < edge[1] && (size_t)l + 2 < n + kTopLevels + 40);
  k_check_ids<<<kSweep, 256, 0, W.st>>>(d_nodes, L.list, d_offsets, n_gauss, st);
  e = cudaGetLastError();
  L.starts.resize((size_t)l + 2);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, st, sizeof h, cudaMemcpyDeviceToHost, W.st);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(L.starts.data(), L.ls, 4 * L.starts.size(), cudaMemcpyDeviceToHost, W.st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(W.st);
  if (e != cudaSuccess) return e;
  L.ok = h.bad == 0;
  L.n = h.tail;
  L.n_leaves = h.n_leaves;
  L.max_leaf = h.max_leaf;
  L.levels = 0;
  while ((size_t)L.levels + 1 < L.starts.size() && L.starts[L.levels] < L.starts[L.levels + 1]) ++L.levels;
  L.top_nodes = L.starts[kTopLevels + 1];
  return cudaSuccess;
}

cudaError_t tree_relayout(WorkMem& W, const uint2* d_nodes, TreeLists& L, uint2* out) {
  uint32_t* sub = W.take<uint32_t>(L.n);
  uint32_t* idx = L.idx = W.take<uint32_t>(L.n);
  uint32_t* pair = W.take<uint32_t>(L.n);
  if (W.err != cudaSuccess) return W.err;
  auto grid = [&](int l) { return std::min(kSweep, blocks_for(L.starts[l + 1] - L.starts[l], 256)); };
  for (int l = L.levels - 1; l >= kTopLevels; --l) k_sums<<<grid(l), 256, 0, W.st>>>(L.cpos, L.ls, l, sub);
  k_place_top<<<1, 1024, 0, W.st>>>(L.cpos, L.ls, sub, idx, pair);
  for (int l = kTopLevels; l < L.levels; ++l) k_place<<<grid(l), 256, 0, W.st>>>(L.cpos, L.ls, sub, l, idx, pair);
  k_relaid<<<blocks_for(L.n, 256), 256, 0, W.st>>>(d_nodes, L.list, L.n, L.cpos, idx, pair, out);
  return cudaGetLastError();
}

cudaError_t tree_leaf_pairs(WorkMem& W, const uint2* relaid, uint32_t n, uint64_t** first, uint64_t* n_pairs) {
  *first = W.take<uint64_t>((size_t)n + 1);
  cudaError_t e = W.err;
  if (e == cudaSuccess) e = scan_of(W, PairOp{relaid, n}, *first, (uint64_t)n + 1);
  if (e == cudaSuccess) e = cudaMemcpyAsync(n_pairs, *first + n, 8, cudaMemcpyDeviceToHost, W.st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(W.st);
  return e;
}

cudaError_t tree_leaf_gids(WorkMem& W, uint2* relaid, uint32_t n, const uint64_t* first, const uint32_t* d_offsets,
                           uint32_t* gid) {
  k_leaf_gids<<<blocks_for(n, 256 / kLeafLanes), 256, 0, W.st>>>(relaid, n, first, d_offsets, gid);
  return cudaGetLastError();
}

cudaError_t tree_leaf_first(WorkMem& W, const TreeLists& L, const uint64_t* first, uint32_t* out) {
  k_leaf_first<<<blocks_for(L.n, 256), 256, 0, W.st>>>(L.list, L.cpos, L.idx, L.n, first, out);
  return cudaGetLastError();
}

cudaError_t aniso_index(WorkMem& W, const uint8_t* flag, uint32_t n, uint32_t** aidx, uint32_t* n_aniso) {
  *aidx = W.take<uint32_t>((size_t)n + 1);
  cudaError_t e = W.err;
  if (e == cudaSuccess) e = scan_of(W, FlagOp{flag, n}, *aidx, (uint64_t)n + 1);
  if (e == cudaSuccess) e = cudaMemcpyAsync(n_aniso, *aidx + n, 4, cudaMemcpyDeviceToHost, W.st);
  if (e != cudaSuccess) return e;
  k_aniso_index<<<blocks_for(n, 256), 256, 0, W.st>>>(flag, n, *aidx);
  return cudaGetLastError();
}

cudaError_t tree_split_counts(WorkMem& W, const uint2* relaid, uint32_t n, const uint32_t* gid, const uint8_t* flag,
                              uint64_t** first, uint64_t* totals) {
  uint64_t* cnt = W.take<uint64_t>((size_t)n + 1);
  *first = W.take<uint64_t>((size_t)n + 1);
  if (W.err != cudaSuccess) return W.err;
  k_split_counts<<<blocks_for((uint64_t)n + 1, 256 / kLeafLanes), 256, 0, W.st>>>(relaid, n, gid, flag, cnt);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = scan_to(W, (const uint64_t*)cnt, *first, (uint64_t)n + 1);
  if (e == cudaSuccess) e = cudaMemcpyAsync(totals, *first + n, 8, cudaMemcpyDeviceToHost, W.st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(W.st);
  return e;
}

cudaError_t tree_split_fill(WorkMem& W, const uint2* relaid, uint32_t n, const uint32_t* gid, const uint8_t* flag,
                            const uint64_t* first, uint2* nodes_p, uint2* aux, uint32_t* gid_plain,
                            uint32_t* gid_flag) {
  k_split_fill<<<blocks_for(n, 256 / kLeafLanes), 256, 0, W.st>>>(relaid, n, gid, flag, first, nodes_p, aux, gid_plain,
                                                                 gid_flag);
  return cudaGetLastError();
}

}  // namespace kdgr
