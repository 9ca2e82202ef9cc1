// Leaf bounding boxes of every node's children, for exact subtree pruning in
// the traversal.
//
// For every node the record holds, per child octet, the box of the leaf
// cells of that child's subtree, relative to the child's cube and rounded
// outward to 1/256 of its edge (8 bits per bound). A ray that misses a
// child's box (expanded by a margin far above the traversal's rounding) can
// reach no leaf of that subtree, so the walk may skip it: the first leaf hit,
// and so every pixel, stays the same, and only the count of nodes visited
// drops.
//
// Record of node i (8 x 8 bytes, one per child octet o): word x = xlo |
// xhi << 8 | ylo << 16 | yhi << 24, word y = zlo | zhi << 8. Bounds
// count cells of 1/256 of the child's edge from the child's x-min, y-max and
// z-max corner (y and z grow downward, as the octet bits do); a bound pair
// lo > hi marks a subtree without leaves.
//
// Levels: the build walks the tree breadth first from the root; the depth of
// the tree is the last level that holds nodes, and the boxes are valid for
// renders whose maxlevel is at least that depth. A node reached twice (not a
// tree: two parents or a cycle, found from each node's position in the
// breadth-first order), a child index outside the array (which the walk
// reports when it meets it) or a tree deeper than the shader's stack leaves
// the boxes unusable.
//
// The level counts stay on the device: every kernel finds its level's range
// from them, and the host reads them once, when all is queued. A node's
// children are neighbours in the order, so their boxes are read in one run,
// and a level's boxes and records are made in one kernel. What bounds it, at
// 0.41 ms of kernels for 2.6M nodes of a 1M-point floor (1.1 with a host wait
// per level, boxes and records in passes of their own): the 64-byte records
// and 32-byte blocks of a level lie scattered (0.3M-0.6M nodes take 20-40 us),
// and 37 launches, most of small levels.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "boxes.cuh"
#include "qbc_internal.h"
#include "qbcuda.h"

using qbc::fail;

namespace qbc {
namespace {

constexpr int kThreads = 256;
constexpr int kLevels = QBC_MAX_LEVEL + 1;  // levels expanded: nodes of a deeper one rule the boxes out

struct Counts {
  unsigned long long level[kLevels + 1];  // nodes per level
  unsigned bad;                           // a child index outside the array, or a node reached twice
};

// First position of level L in the order, and its end.
__device__ __forceinline__ void level_range(const Counts* c, int L, int64_t* b, int64_t* e) {
  unsigned long long at = 0;
  for (int k = 0; k < L; ++k) at += c->level[k];
  *b = (int64_t)at;
  *e = (int64_t)(at + c->level[L]);
}

// Children of the nodes of level L appended to the order after them, each
// with its position in pos; a node's first child's position to `first`. One
// counter update per block and pass: each thread takes its node's children,
// the block reserves their total at once (one update per warp: 38 us for a
// level of 0.6M nodes, the updates of one address in turn; 25 so).
__global__ void __launch_bounds__(kThreads) expand_kernel(const int4* __restrict__ child, int64_t n,
                                                          int32_t* __restrict__ order, int32_t* __restrict__ pos,
                                                          int32_t* __restrict__ first, Counts* counts, int L) {
  __shared__ unsigned warp_total[kThreads / 32];
  __shared__ unsigned long long reserved;
  int64_t in_b, in_e;
  level_range(counts, L, &in_b, &in_e);
  if (in_e > n) return;  // not a tree, detected on the host
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  // the loop's trip count is the same for the whole block (barriers below)
  for (int64_t j0 = in_b + blockIdx.x * (int64_t)kThreads; j0 < in_e; j0 += stride) {
    const int64_t j = j0 + tid;
    int32_t c[8];
    uint32_t take = 0;
    bool outside = false;
    if (j < in_e) {
      load_children(child, order[j], c);
#pragma unroll
      for (int o = 0; o < 8; ++o) {
        take |= (c[o] > 0 && c[o] < n) ? (1u << o) : 0u;
        // an index outside the array: the walk must meet it (it reports
        // it), so no boxes for this tree
        outside |= c[o] != 0 && !(c[o] > 0 && c[o] < n);
      }
    }
    if (__any_sync(0xFFFFFFFFu, outside) && lane == 0) counts->bad = 1u;
    const unsigned mine = (unsigned)__popc(take);
    unsigned incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) warp_total[warp] = incl;
    __syncthreads();
    unsigned before = incl - mine, total = 0;
#pragma unroll
    for (int k = 0; k < kThreads / 32; ++k) {
      if (k < warp) before += warp_total[k];
      total += warp_total[k];
    }
    if (tid == 0) reserved = total ? atomicAdd(&counts->level[L + 1], (unsigned long long)total) : 0ull;
    __syncthreads();
    int64_t k = in_e + (int64_t)reserved + before;
    if (j < in_e) first[j] = (int32_t)min(k, n);
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      if ((take >> o) & 1u) {
        if (k < n) {  // past n: not a tree, detected on the host
          order[k] = c[o];
          pos[c[o]] = (int32_t)k;
        }
        ++k;
      }
    }
  }
}

// A node appended twice (two parents, or a cycle) keeps one of its positions
// in pos, so another position of it disagrees: then the array is not a tree.
__global__ void unique_kernel(const int32_t* __restrict__ order, const int32_t* __restrict__ pos, int64_t n,
                              Counts* counts) {
  int64_t b, e;
  level_range(counts, kLevels, &b, &e);
  if (e > n) return;
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < e; j += (int64_t)gridDim.x * blockDim.x)
    if (pos[order[j]] != (int32_t)j) counts->bad = 1u;
}

// Boxes in leaf cells of the nodes of level L, by position (children done),
// and their records.
__global__ void __launch_bounds__(kThreads)
    box_level_kernel(const int4* __restrict__ child, int64_t n, const int32_t* __restrict__ order,
                     const int32_t* __restrict__ first, const Counts* counts, int L, uint4* __restrict__ box,
                     uint4* __restrict__ rec) {
  int64_t b, e, all_b, all_e;
  level_range(counts, L, &b, &e);
  level_range(counts, kLevels, &all_b, &all_e);
  if (counts->bad || all_e > n || all_b < all_e) return;  // no boxes
  int depth = L;
  while (depth + 1 <= kLevels && counts->level[depth + 1] > 0) ++depth;
  if (L == depth) return;  // leaf cells: their box is their own cell
  const bool last = L + 1 == depth;
  const int sh = depth - L - 1;  // a child's edge: 2^sh leaf cells
  for (int64_t j = b + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < e; j += (int64_t)gridDim.x * blockDim.x) {
    const int32_t node = order[j];
    int32_t c[8];
    load_children(child, node, c);
    const int64_t k = first[j];
    // all children's boxes are read before the first is used (they depend on
    // nothing but their number)
    uint4 raw[8];
    int m = 0;
#pragma unroll
    for (int o = 0; o < 8; ++o)
      if (c[o] > 0 && c[o] < n) raw[o] = last ? make_uint4(0u, 0u, 0u, 0u) : box[k + m++];
    CellBox u = no_box();
    uint2 w[8];
#pragma unroll
    for (int o = 0; o < 8; ++o) {
      w[o] = empty_word();
      if (!(c[o] > 0 && c[o] < n)) continue;
      const CellBox v = unpack_box(raw[o]);
      if (v.lo[0] > v.hi[0]) continue;  // no leaves below
      w[o] = record_word(v, sh);
      add_box(u, v, o, sh);
    }
    box[j] = pack_box(u);
    store_record(rec, node, w);
  }
}

}  // namespace

size_t box_scratch(int64_t n) { return (size_t)n * 28 + sizeof(Counts) + 64; }

int build_child_boxes(const int32_t* child, int64_t n, uint32_t* rec, void* scratch, cudaStream_t stream, int grid,
                      int* depth, int64_t* launches) {
  *depth = -1;
  if (n <= 0) return QBC_OK;
  uint4* box = static_cast<uint4*>(scratch);
  int32_t* order = reinterpret_cast<int32_t*>(box + n);
  int32_t* pos = order + n;
  int32_t* first = pos + n;
  Counts* counts =
      reinterpret_cast<Counts*>((reinterpret_cast<uintptr_t>(first + n) + 15) & ~static_cast<uintptr_t>(15));
  const int4* blocks = reinterpret_cast<const int4*>(child);
  uint4* records = reinterpret_cast<uint4*>(rec);
  const unsigned long long one = 1;
  cudaError_t e = cudaMemsetAsync(counts, 0, sizeof(Counts), stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&counts->level[0], &one, 8, cudaMemcpyHostToDevice, stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(order, 0, 4, stream);  // the root
  if (e == cudaSuccess) e = cudaMemsetAsync(pos, 0, 4, stream);
  if (e != cudaSuccess) return fail(QBC_E_CUDA, "box build: %s", cudaGetErrorString(e));
  // blocks of a level's kernel: the level holds at most min(n, 8^L) nodes
  auto blocks_of = [&](int L) {
    const int64_t most = L >= 10 ? n : std::min<int64_t>(n, int64_t(1) << (3 * L));
    return (unsigned)std::min<int64_t>(grid, (most + kThreads - 1) / kThreads);
  };
  for (int L = 0; L < kLevels; ++L)
    expand_kernel<<<blocks_of(L), kThreads, 0, stream>>>(blocks, n, order, pos, first, counts, L);
  unique_kernel<<<blocks_of(kLevels), kThreads, 0, stream>>>(order, pos, n, counts);
  for (int L = kLevels - 1; L >= 0; --L)
    box_level_kernel<<<blocks_of(L), kThreads, 0, stream>>>(blocks, n, order, first, counts, L, box, records);
  *launches += 2 * kLevels + 1;
  Counts h;
  e = cudaMemcpyAsync(&h, counts, sizeof(h), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return fail(QBC_E_CUDA, "box build: %s", cudaGetErrorString(e));
  unsigned long long total = 0;
  for (int L = 0; L <= kLevels; ++L) total += h.level[L];
  if (h.bad || (int64_t)total > n || h.level[kLevels] > 0) return QBC_OK;  // no boxes
  int D = 0;
  while (h.level[D + 1] > 0) ++D;
  *depth = D;
  return QBC_OK;
}

}  // namespace qbc
