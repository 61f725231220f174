// Connected components on the device (find_components, src/components.rs:7-44).
//
// Lock-free union-find: every edge hooks the larger of its two roots under
// the smaller one with atomicCAS, so parent[x] <= x always holds and the final
// root of a component is its smallest node.  Numbering components by the rank
// of their root therefore reproduces the crate's BFS labels (components are
// numbered in the order of their smallest node) for symmetric graphs.  Every
// loop is bounded: a failed CAS means some root was hooked to a strictly
// smaller node, and root chains only shrink.
#include <cub/cub.cuh>

#include "si_internal.h"

namespace si {
namespace {

__device__ __forceinline__ uint32_t find_root(uint32_t* parent, uint32_t x) {
  // path halving; parents only ever decrease, so the benign races are safe
  for (int guard = 0; guard < (1 << 30); ++guard) {
    const uint32_t p = parent[x];
    if (p == x) return x;
    const uint32_t gp = parent[p];
    if (gp != p) parent[x] = gp;
    x = gp;
  }
  return x;
}

// A row starts under its first neighbour when that is smaller (parents always
// are: no cycles), which already joins most of a kNN graph.
__global__ void k_init_parent(int64_t n, const uint64_t* __restrict__ indptr, const uint32_t* __restrict__ indices,
                              uint32_t* parent) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n; i += stride) {
    uint32_t p = static_cast<uint32_t>(i);
    if (indptr[i] < indptr[i + 1]) p = min(p, indices[indptr[i]]);
    parent[i] = p;
  }
}

__device__ __forceinline__ void unite(uint32_t* parent, uint32_t a, uint32_t b) {
  uint32_t ri = find_root(parent, a), rj = find_root(parent, b);
  for (int guard = 0; guard < (1 << 30) && ri != rj; ++guard) {
    const uint32_t hi = ri > rj ? ri : rj;
    const uint32_t lo = ri > rj ? rj : ri;
    const uint32_t old = atomicCAS(parent + hi, hi, lo);
    if (old == hi) break;
    ri = find_root(parent, old);
    rj = find_root(parent, lo);
  }
}

// One more edge of every row, its last: with the first, two edges a node leave
// nearly all of a kNN graph in one tree (the sampling of Sutton, Ben-Nun and
// Barak, "Optimizing parallel graph connectivity computation via subgraph
// sampling", IPDPS 2018).
__global__ void k_hook_last(int64_t n, const uint64_t* __restrict__ indptr, const uint32_t* __restrict__ indices,
                            uint32_t* parent) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n; i += stride)
    if (indptr[i] < indptr[i + 1]) unite(parent, static_cast<uint32_t>(i), indices[indptr[i + 1] - 1]);
}

// The remaining edges, eight lanes a row: after a compression, ends with the
// same parent are in one tree, which settles nearly every edge with one load.
// Uniting along every edge, a thread a row, took 790 us at n = 200k.
__global__ void k_hook(int64_t n, const uint64_t* __restrict__ indptr, const uint32_t* __restrict__ indices,
                       uint32_t* parent) {
  const int sub = threadIdx.x & 7;
  const int64_t groups = static_cast<int64_t>(gridDim.x) * blockDim.x / 8;
  for (int64_t i = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) / 8; i < n; i += groups) {
    const uint32_t pi = parent[i];
    for (uint64_t k = indptr[i] + sub; k < indptr[i + 1]; k += 8) {
      const uint32_t j = indices[k];
      if (parent[j] != pi) unite(parent, static_cast<uint32_t>(i), j);
    }
  }
}

// Every node under its root, a thread a node.  Only a node's own thread writes
// its parent (path halving here let one thread put a stale inner node over the
// root that another had found), and it writes every step: nodes of one chain in
// flight together jump over one another, so a chain of length l takes about
// log l steps.  That wants the smaller nodes, where parents lie, in flight or
// done: blocks start in order, and there is no second node for a thread, whose
// chain would lead through blocks that have not started (a path of 1M nodes in
// order took 55 ms so and takes 0.2 now; with path halving it took 40).
__global__ void k_compress(int64_t n, uint32_t* parent, uint32_t* is_root) {
  const int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  uint32_t r = __ldcg(parent + i);
  is_root[i] = (r == static_cast<uint32_t>(i)) ? 1u : 0u;
  for (uint32_t p = __ldcg(parent + r); p != r; p = __ldcg(parent + r)) {  // parents decrease
    r = p;
    __stcg(parent + i, r);
  }
}

__global__ void k_label(int64_t n, const uint32_t* __restrict__ parent, const uint32_t* __restrict__ rank,
                        uint32_t* __restrict__ labels) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n; i += stride)
    labels[i] = rank[parent[i]];
}

}  // namespace

int64_t find_components_dev(const Exec& ex, const GraphDev& g, uint32_t* labels) {
  if (g.n == 0) return 0;
  const int threads = 256;
  const int grid = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((g.n + threads - 1) / threads,
                                                                           int64_t(ex.sms) * 16)));
  const unsigned nodes = static_cast<unsigned>((g.n + threads - 1) / threads);
  DevBuf<uint32_t> parent(g.n, ex.stream), is_root(g.n + 1, ex.stream), rank(g.n + 1, ex.stream);
  k_init_parent<<<grid, threads, 0, ex.stream>>>(g.n, g.indptr, g.indices, parent.get());
  SI_LAUNCH_CHECK();
  k_compress<<<nodes, threads, 0, ex.stream>>>(g.n, parent.get(), is_root.get());
  SI_LAUNCH_CHECK();
  k_hook_last<<<grid, threads, 0, ex.stream>>>(g.n, g.indptr, g.indices, parent.get());
  SI_LAUNCH_CHECK();
  k_compress<<<nodes, threads, 0, ex.stream>>>(g.n, parent.get(), is_root.get());
  SI_LAUNCH_CHECK();
  const int hook_grid = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>((g.n * 8 + threads - 1) / threads,
                                                                                int64_t(ex.sms) * 16)));
  k_hook<<<hook_grid, threads, 0, ex.stream>>>(g.n, g.indptr, g.indices, parent.get());
  SI_LAUNCH_CHECK();
  SI_CUDA(cudaMemsetAsync(is_root.get() + g.n, 0, sizeof(uint32_t), ex.stream));
  k_compress<<<nodes, threads, 0, ex.stream>>>(g.n, parent.get(), is_root.get());
  SI_LAUNCH_CHECK();
  size_t tmp_bytes = 0;
  SI_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, is_root.get(), rank.get(), g.n + 1, ex.stream));
  DevBuf<unsigned char> tmp(tmp_bytes, ex.stream);
  SI_CUDA(cub::DeviceScan::ExclusiveSum(tmp.get(), tmp_bytes, is_root.get(), rank.get(), g.n + 1, ex.stream));
  k_label<<<grid, threads, 0, ex.stream>>>(g.n, parent.get(), rank.get(), labels);
  SI_LAUNCH_CHECK();
  uint32_t total = 0;
  SI_CUDA(cudaMemcpyAsync(&total, rank.get() + g.n, sizeof(uint32_t), cudaMemcpyDeviceToHost, ex.stream));
  SI_CUDA(cudaStreamSynchronize(ex.stream));
  return static_cast<int64_t>(total);
}

}  // namespace si
