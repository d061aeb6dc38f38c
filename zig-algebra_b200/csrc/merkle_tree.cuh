// merkle_tree.cuh -- heap-ordered BLAKE3 Merkle trees on the device, the
// layout of MerkleTree (libs/merkle/src/merkle_tree.zig:70-180): node 1 the
// root, node w + j entry j of the level of width w, node i the hash of nodes
// 2i and 2i + 1, node 0 zero.  A leaf source (layer pairs, folded pairs,
// rows, or digests of an earlier launch) supplies the bottom level.
//
// The tree is built bottom-up in subtrees: a thread hashes two siblings and
// their parent in registers, and a CTA of 256 threads takes its 256 parents
// three levels further through shared memory, where every level still fills
// whole warps: five levels a subtree.  A commitment whose caller waits for the
// root runs all subtrees in one launch (tree_kernel), the others one launch per
// four or five levels.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "blake3.cuh"
#include "runtime.hpp"

namespace zntt {

namespace {

constexpr int kThreads = 256;     // CTA size of the subtree kernels
constexpr int kSharedLevels = 3;  // levels a CTA builds in shared memory (256 -> 32 nodes)

__device__ __forceinline__ void store_digest(uint4* nodes, uint64_t i, const uint32_t (&d)[8]) {
  nodes[2 * i] = make_uint4(d[0], d[1], d[2], d[3]);
  nodes[2 * i + 1] = make_uint4(d[4], d[5], d[6], d[7]);
}

__device__ __forceinline__ void load_digest(const uint4* nodes, uint64_t i, uint32_t (&d)[8]) {
  const uint4 a = nodes[2 * i], b = nodes[2 * i + 1];
  d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w;
  d[4] = b.x; d[5] = b.y; d[6] = b.z; d[7] = b.w;
}

// The same from nodes that other CTAs of the launch wrote.
__device__ __forceinline__ void load_digest_cg(const uint4* nodes, uint64_t i, uint32_t (&d)[8]) {
  const uint4 a = __ldcg(nodes + 2 * i), b = __ldcg(nodes + 2 * i + 1);
  d[0] = a.x; d[1] = a.y; d[2] = a.z; d[3] = a.w;
  d[4] = b.x; d[5] = b.y; d[6] = b.z; d[7] = b.w;
}

// Source of a subtree's bottom level.  Leaf sources hash pairs of layer
// values; the node source reads digests an earlier launch wrote.
struct NodeSource {
  const uint4* nodes;
  uint64_t width;  // the level read: nodes [width, 2 width)
  __device__ __forceinline__ void get(uint64_t j, uint32_t (&d)[8], uint32_t) const {
    load_digest_cg(nodes, width + j, d);
  }
};
// Every leaf j < h on its own (small trees).
template <class Src>
__global__ void leaf_kernel(Src src, uint4* __restrict__ nodes, uint64_t h, uint32_t one) {
  for (uint64_t j = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; j < h; j += (uint64_t)gridDim.x * blockDim.x) {
    uint32_t d[8];
    src.get(j, d, one);
    store_digest(nodes, h + j, d);
  }
}

// The digests a CTA passes from level to level.
struct TreeShared {
  uint4 a[kThreads][2], b[kThreads / 2][2];
};

// `levels` levels above the cnt digests in sm.a, stored from node `first_node`
// of the first one on: level l has cnt >> l nodes of this CTA, the first of them
// node (first_node >> l).  Ends with a barrier.
__device__ __forceinline__ void shared_levels(TreeShared& sm, uint4* nodes, uint64_t first_node, uint32_t cnt,
                                              int levels, uint32_t one) {
  const uint32_t t = threadIdx.x;
  uint4(*from)[2] = sm.a;
  uint4(*to)[2] = sm.b;
#pragma unroll 1
  for (int lev = 1; lev <= levels; lev++) {
    cnt >>= 1;
    first_node >>= 1;
    if (t < cnt) {
      const uint4 a0 = from[2 * t][0], a1 = from[2 * t][1], b0 = from[2 * t + 1][0], b1 = from[2 * t + 1][1];
      const uint32_t m[16] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w,
                              b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
      uint32_t d[8];
      b3_hash_block<true>(m, 64, d, one);
      store_digest(nodes, first_node + t, d);
      if (lev < levels) {
        to[t][0] = make_uint4(d[0], d[1], d[2], d[3]);
        to[t][1] = make_uint4(d[4], d[5], d[6], d[7]);
      }
    }
    __syncthreads();
    uint4(*x)[2] = from;
    from = to;
    to = x;
  }
}

// Subtree `blk` over the level of width w (a multiple of 512): thread t takes
// entries 2u and 2u + 1 of that level (u = 256 blk + t), hashes their parent in
// registers, and the CTA builds three more levels in shared memory, each still
// whole warps (128, 64, 32 nodes).  Writes the levels of width w/2 .. w/16, and
// the bottom level itself when it is made here (leaves).
template <class Src, bool kStoreBottom>
__device__ __forceinline__ void subtree(const Src& src, uint4* nodes, uint64_t w, uint64_t blk, uint32_t one,
                                        TreeShared& sm) {
  const uint32_t t = threadIdx.x;
  const uint64_t u = blk * kThreads + t;
  uint32_t l[8], r[8], p[8];
  src.get(2 * u, l, one);
  if (kStoreBottom) store_digest(nodes, w + 2 * u, l);
  src.get(2 * u + 1, r, one);
  if (kStoreBottom) store_digest(nodes, w + 2 * u + 1, r);
  b3_parent(l, r, p, one);
  store_digest(nodes, (w >> 1) + u, p);
  sm.a[t][0] = make_uint4(p[0], p[1], p[2], p[3]);
  sm.a[t][1] = make_uint4(p[4], p[5], p[6], p[7]);
  __syncthreads();
  shared_levels(sm, nodes, (w >> 1) + blk * kThreads, kThreads, kSharedLevels, one);
}

template <class Src, bool kStoreBottom>
__global__ void __launch_bounds__(kThreads) subtree_kernel(Src src, uint4* __restrict__ nodes, uint64_t w,
                                                           uint32_t one) {
  __shared__ TreeShared sm;
  subtree<Src, kStoreBottom>(src, nodes, w, blockIdx.x, one, sm);
}

// Where a synchronous commitment delivers its root: pinned host memory that the
// kernel writes, the sequence number last.
struct RootOut {
  uint4* root;
  volatile uint32_t* seq;
  uint32_t value;
};

// The rest of the tree above the w <= 256 digests in sm.a (level w, already in
// `nodes`), then node 0 and the root for the host.
__device__ __forceinline__ void finish_tree(TreeShared& sm, uint4* nodes, uint32_t w, const RootOut& out,
                                            uint32_t one) {
  shared_levels(sm, nodes, w, w, 31 - __clz(w), one);
  if (threadIdx.x == 0) {
    nodes[0] = nodes[1] = make_uint4(0, 0, 0, 0);  // node 0 is unused and zero
    out.root[0] = nodes[2];
    out.root[1] = nodes[3];
    __threadfence_system();
    *out.seq = out.value;
  }
}

// A whole tree over the level of width w (a multiple of 512) in one launch: CTA
// b builds its subtree, and the last CTA of each sixteen to finish goes on with
// the next one, over the 512 nodes those sixteen wrote (counted by `tickets`,
// which each last CTA sets back to zero); the last of all builds the top.  No
// CTA waits for another.  Against a launch per four levels and one for the top
// this saves the launches between, most of a small tree's time.
template <class Src, bool kStoreBottom>
__global__ void __launch_bounds__(kThreads) tree_kernel(Src src, uint4* nodes, uint64_t w, uint32_t* tickets,
                                                        RootOut out, uint32_t one) {
  __shared__ TreeShared sm;
  __shared__ bool s_last;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  uint64_t blk = blockIdx.x, groups = gridDim.x;
  subtree<Src, kStoreBottom>(src, nodes, w, blk, one, sm);
  for (;;) {
    w >>= 1 + kSharedLevels;  // 32 nodes of this CTA
    const uint32_t size = groups < 16 ? (uint32_t)groups : 16u;
    blk /= size;
    groups /= size;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      s_last = atomicAdd(&tickets[blk], 1u) == size - 1;
      if (s_last) tickets[blk] = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    tickets += groups;
    if (w < 2 * kThreads) break;
    subtree<NodeSource, false>(NodeSource{nodes, w}, nodes, w, blk, one, sm);
  }
  if (threadIdx.x < w) {
    uint32_t d[8];
    load_digest_cg(nodes, w + threadIdx.x, d);
    sm.a[threadIdx.x][0] = make_uint4(d[0], d[1], d[2], d[3]);
    sm.a[threadIdx.x][1] = make_uint4(d[4], d[5], d[6], d[7]);
  }
  __syncthreads();
  finish_tree(sm, nodes, (uint32_t)w, out, one);
}

// A tree of h <= 256 leaves in one CTA.
template <class Src>
__global__ void __launch_bounds__(kThreads) small_tree_kernel(Src src, uint4* nodes, uint32_t h, RootOut out,
                                                              uint32_t one) {
  __shared__ TreeShared sm;
  const uint32_t t = threadIdx.x;
  if (t < h) {
    uint32_t d[8];
    src.get(t, d, one);
    store_digest(nodes, h + t, d);
    sm.a[t][0] = make_uint4(d[0], d[1], d[2], d[3]);
    sm.a[t][1] = make_uint4(d[4], d[5], d[6], d[7]);
  }
  __syncthreads();
  finish_tree(sm, nodes, h, out, one);
}

// The levels of width w_top, w_top / 2, ..., 1 in one CTA; the barrier between
// levels orders each level's global writes before the next level's reads.
__global__ void top_levels_kernel(uint4* nodes, uint32_t w_top, uint32_t one) {
  for (uint32_t w = w_top; w >= 1; w >>= 1) {
    for (uint32_t i = threadIdx.x; i < w; i += blockDim.x) {
      uint32_t l[8], r[8], d[8];
      load_digest(nodes, 2 * ((uint64_t)w + i), l);
      load_digest(nodes, 2 * ((uint64_t)w + i) + 1, r);
      b3_parent(l, r, d, one);
      store_digest(nodes, (uint64_t)w + i, d);
    }
    __syncthreads();
  }
}

int grid_for_count(uint64_t count) { return (int)std::min<uint64_t>((count + 255) / 256, 148 * 16); }

// Sources whose leaves are costly enough to run one per thread in leaf_kernel
// specialize this to true.
template <class T>
struct OneLeafPerThread {
  static constexpr bool value = false;
};

// Leaves, then subtrees while a level has 512 entries or more (each launch four
// new levels, five where it makes the leaves too), then the rest in one CTA: the launches of a commitment that the caller does
// not wait for (it may be captured, or run beside others).
template <class Src>
cudaError_t build_tree(const Src& src, uint4* nodes, uint64_t h, cudaStream_t st) {
  uint64_t w = h;
  if (h >= 2 * kThreads && !OneLeafPerThread<Src>::value) {
    subtree_kernel<Src, true><<<(unsigned)(h / (2 * kThreads)), kThreads, 0, st>>>(src, nodes, h, 1u);
    w = h >> (1 + kSharedLevels);
  } else {
    leaf_kernel<Src><<<grid_for_count(h), kThreads, 0, st>>>(src, nodes, h, 1u);
  }
  cudaError_t ce = cudaGetLastError();
  for (; w >= 2 * kThreads && ce == cudaSuccess; w >>= 1 + kSharedLevels) {
    subtree_kernel<NodeSource, false><<<(unsigned)(w / (2 * kThreads)), kThreads, 0, st>>>(NodeSource{nodes, w},
                                                                                           nodes, w, 1u);
    ce = cudaGetLastError();
  }
  if (w >= 2 && ce == cudaSuccess) {
    top_levels_kernel<<<1, 1024, 0, st>>>(nodes, (uint32_t)(w / 2), 1u);
    ce = cudaGetLastError();
  }
  return ce;
}

// Levels of at least this width get launches of their own, one per four new levels
// (five where the leaves are made too):
// with as many CTAs the fences and counts of tree_kernel cost more than launches
// save.  A Goldilocks layer and its root, one launch against this line: 2^18 42.5
// and 41 us, 2^20 72 and 67, 2^24 560 and 516; below it one launch is the faster
// (2^16 33.9 us, 43.5 in launches; lines at 2^19 and 2^21 are no faster; B200).
constexpr uint64_t kOwnLaunchWidth = (uint64_t)1 << 17;
// So a tree_kernel's level has at most half of that, 128 subtrees in groups of sixteen: 8
// counters for the first level of groups and one for the last.
static_assert(kOwnLaunchWidth / 2 / (2 * kThreads) <= 256 && 256 / 16 + 1 <= kTreeTickets, "a counter for every group");

// tree_kernel over the level of width w, made by the launch before it on `st`.
cudaError_t launch_node_tree(uint4* nodes, uint64_t w, uint32_t* tickets, const RootOut& out, cudaStream_t st) {
  for (; w >= kOwnLaunchWidth; w >>= 1 + kSharedLevels) {
    subtree_kernel<NodeSource, false><<<(unsigned)(w / (2 * kThreads)), kThreads, 0, st>>>(NodeSource{nodes, w},
                                                                                           nodes, w, 1u);
    const cudaError_t ce = cudaGetLastError();
    if (ce != cudaSuccess) return ce;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(w / (2 * kThreads)));
  cfg.blockDim = dim3(kThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, tree_kernel<NodeSource, false>, NodeSource{nodes, w}, nodes, w, tickets, out, 1u);
}

// The same tree for a caller that waits for its root: one launch where it is not
// wide (after one for leaves that run one per thread), which delivers the root.
template <class Src>
cudaError_t build_tree_root(const Src& src, uint4* nodes, uint64_t h, uint32_t* tickets, const RootOut& out,
                            cudaStream_t st) {
  if (h <= kThreads) {
    small_tree_kernel<Src><<<1, kThreads, 0, st>>>(src, nodes, (uint32_t)h, out, 1u);
    return cudaGetLastError();
  }
  if (OneLeafPerThread<Src>::value) {
    // Few leaves: small CTAs, so that they spread over the SMs.
    const uint32_t threads = h <= 148 * 256 ? 64 : kThreads;
    leaf_kernel<Src><<<(unsigned)std::min<uint64_t>(h / threads, 148 * 16), threads, 0, st>>>(src, nodes, h, 1u);
    const cudaError_t ce = cudaGetLastError();
    return ce == cudaSuccess ? launch_node_tree(nodes, h, tickets, out, st) : ce;
  }
  const unsigned grid = (unsigned)(h / (2 * kThreads));
  if (h >= kOwnLaunchWidth) {
    subtree_kernel<Src, true><<<grid, kThreads, 0, st>>>(src, nodes, h, 1u);
    const cudaError_t ce = cudaGetLastError();
    return ce == cudaSuccess ? launch_node_tree(nodes, h >> (1 + kSharedLevels), tickets, out, st) : ce;
  }
  tree_kernel<Src, true><<<grid, kThreads, 0, st>>>(src, nodes, h, tickets, out, 1u);
  return cudaGetLastError();
}

// A commitment over h leaves on `st`.  With root_out it returns once the root is
// there (and with it every node), or with `settle` once the stream has retired
// the work.  Without root_out it only enqueues.
template <class Src>
int commit_tree(const Src& src, uint4* nodes, uint64_t h, uint8_t* root_out, cudaStream_t st, bool settle, const char* what) {
  if (!root_out) {
    cudaError_t ce = cudaMemsetAsync(nodes, 0, 32, st);  // node 0 is unused and zero
    if (ce == cudaSuccess) ce = build_tree(src, nodes, h, st);
    return ce == cudaSuccess ? ZNTT_OK : cuda_fail(ce, what);
  }
  RootWait wait;
  int rc = root_wait_begin(&wait);
  if (rc) return rc;
  const cudaError_t ce =
      build_tree_root(src, nodes, h, wait.tickets, RootOut{static_cast<uint4*>(wait.root), wait.seq, wait.value}, st);
  if (ce != cudaSuccess) return cuda_fail(ce, what);
  rc = root_wait(wait, st, root_out, what);
  if (rc || !settle) return rc;
  const cudaError_t se = cudaStreamSynchronize(st);
  return se == cudaSuccess ? ZNTT_OK : cuda_fail(se, what);
}

}  // namespace

}  // namespace zntt
