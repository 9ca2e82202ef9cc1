// GPU node-array builder: the same node array as inserting points one by one
// with octree_insert_point (src/qubatron/octree.c:95-147) or octet paths with
// octree_insert_path (octree.c:149-180) into an empty tree, numbering
// included, without the sequential walk, without sorting and without any host
// round trip, so that a per-frame rebuild can be captured in a CUDA graph.
//
// Sequential insertion appends a node the first time a path prefix appears:
// point i walks down the nodes earlier points made and appends the rest of
// its path. So the node of a level-l prefix is created by the smallest point
// index having that prefix (its "creator"), and point i creates exactly the
// levels [c_i, levels] where c_i is the first level whose node it creates.
// Node ids follow from one prefix sum over points in index order:
//   id(i, l) = 1 + sum_{j < i} (levels - c_j + 1) + (l - c_i).
//
// Creators, level by level: the level-l group of a point is (creator of its
// level-(l-1) node, its level-l octet), a slot creator * 8 + octet of a table
// the points atomicMin their index into; the next kernel reads the winner. A
// run of lanes with one slot proposes once (its first lane holds its
// minimum), and only where the table's value is larger. The top levels use
// tables indexed by the prefix itself, all filled by the kernel that makes
// the keys, reduced in shared memory per block. The deeper levels rotate
// three tables of 8 entries per point; a level's winners reset its entries
// two kernels later, so the tables are empty again when the build ends.
//
// A point's nodes have consecutive ids, each the child of the one before, so
// spread_kernel writes their child blocks whole and only the first node of a
// point is linked into its parent (link_kernel).
//
// Leaf boxes: climb_kernel starts at every leaf and goes up: a node with one
// child takes its box shifted; at a node with more, all but the last arriving
// child's thread stop, and the last, whose siblings' boxes are written by
// then, makes the union. Each node's record holds its children's boxes
// quantised outward to 1/256 of a child's edge, the format the render
// kernels' pruning reads (boxes.cu builds the same records for uploaded
// trees). No thread waits: a thread that is not last ends.
//
// Points given in path order (as assets are) need no creator tables: a point
// creates the levels below the prefix it shares with the point before it, and
// the creator of a prefix is the first point of its run, found by a
// galloping search. A static build, which waits for its node count anyway,
// looks at the order first.
//
// What bounds it: 20M points of a room nearly in path order, 52M nodes, take
// 4.8 ms of kernels (climb 2.1, its chain of dependent loads; tables 1.7, L2
// atomics; blocks 0.4; keys 0.3) and 0.4 of allocations, where writing the
// nodes and records alone, 5.2 GB, takes 0.8. Boxes by a pass over all points
// per level took 7.7 ms, by one pass a level over nodes 3.2.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>
#include <vector>

#include "boxes.cuh"
#include "qbc_internal.h"
#include "qbcuda.h"

using qbc::fail;

namespace qbc {
namespace {

constexpr int kMaxBuildLevels = 21;   // 3 bits per level in a 64-bit key
constexpr int kDense = 4;             // levels 1..kDense use prefix-indexed tables
constexpr int kDenseEntries = 8 + 64 + 512 + 4096;
constexpr uint64_t kExcluded = ~0ull;  // key of a point left out (bad input)
constexpr uint32_t kNone = 0xFFFFFFFFu;
// Points in any order (a character's) crowd at the top tables' few entries:
// 2M points on 200 to 3000 entries spent 500 us on levels 5 to 8, half of a
// build, on atomics to entries that nothing had reached yet and on reads of
// the same few L2 sectors. So a first launch lets kPilot points propose, and
// the others, which mostly find a smaller index then, read the entry through
// their SM's own cache (a copy from before the launch would be stale for
// good). 2M points built, skinned and drawn: 5.33 -> 5.12 ms; with 2048, 32768
// and 131072 pilot points 5.13, 5.13 and 5.18; on all levels 5.13. At 50k
// points the extra launches cost 3 us and gain nothing; points of static
// trees mostly lie in path order, where they cost 0.6 %.
constexpr int64_t kPilot = 8192, kPilotMin = 262144;
constexpr int kPilotLevel = 9;
constexpr int kKeyGroups = 4;         // groups of 32 points a warp makes keys of at a time
constexpr int kClimbThreads = 64;      // threads end at different levels: small blocks give their room back early
// Points per chunk of the prefix sum and of the child blocks' writing: 8 a
// thread, and 1 up to kScanFew points (still one pass over the chunk sums),
// whose few chunks left most SMs idle and each warp a long run of blocks: 50k
// points 50 us for the two kernels in 25 chunks, 13 in 196; a 50k-point
// character skinned, built and drawn 798 -> 788 us.
constexpr int kScanThreads = 256, kScanPer = 8;
constexpr int64_t kScanFew = 262144;

constexpr int64_t scan_chunks(int64_t n) {
  const int64_t chunk = kScanThreads * (n <= kScanFew ? 1 : kScanPer);
  return n <= 0 ? 1 : (n + chunk - 1) / chunk;
}
// ... of any build of at most n points.
constexpr int64_t scan_chunks_most(int64_t n) {
  return n <= kScanFew ? scan_chunks(n) : std::max(scan_chunks(n), scan_chunks(kScanFew));
}

__host__ __device__ constexpr int dense_offset(int l) {  // first entry of level l's prefix table
  return l <= 1 ? 0 : (l == 2 ? 8 : (l == 3 ? 72 : 584));
}

// The low 21 bits of v, one every third bit.
__device__ __forceinline__ uint64_t spread3(uint32_t v) {
  uint64_t x = v & 0x1FFFFFu;
  x = (x | (x << 32)) & 0x001F00000000FFFFull;
  x = (x | (x << 16)) & 0x001F0000FF0000FFull;
  x = (x | (x << 8)) & 0x100F00F00F00F00Full;
  x = (x | (x << 4)) & 0x10C30C30C30C30C3ull;
  x = (x | (x << 2)) & 0x1249249249249249ull;
  return x;
}

// Path key of point i (octets of octree.c:100-109 for points: size halves
// from the basecube edge, (int)(x / size) % 2 picks the x bit, y and z below
// the midline set bits 1 and 2; or the given octets); false for a bad one.
// Halving is exact for a basecube edge that is far from denormal, so x / size
// is x / (edge / 2) times a power of two, and the bits of all levels are
// those of one integer: 3 divisions a point instead of 3 a level.
__device__ __forceinline__ bool path_key(const float* __restrict__ pts, const int32_t* __restrict__ octets, int64_t i,
                                         float basesize, int levels, uint64_t* key) {
  uint64_t k = 0;
  bool ok = true;
  if (pts) {
    const float x = pts[3 * i], y = pts[3 * i + 1], z = pts[3 * i + 2];
    if (!(x >= 0.0f && x < 1.0e30f && y >= 0.0f && y < 1.0e30f && z >= 0.0f && z < 1.0e30f)) {
      ok = false;
    } else if (levels > 0) {
      const float half = basesize / 2.0f, deep = __int_as_float((126 + levels) << 23);  // 2^(levels - 1)
      const float qx = (x / half) * deep, qy = (y / half) * deep, qz = (z / half) * deep;
      if (basesize > 1.0e-20f && fmaxf(fmaxf(qx, qy), qz) < 2147483648.0f) {
        const uint32_t all = (1u << levels) - 1u;
        k = spread3((uint32_t)qx & all) | (spread3(~(uint32_t)qy & all) << 1) | (spread3(~(uint32_t)qz & all) << 2);
      } else {
        float size = basesize;
        for (int level = 0; level < levels; ++level) {
          size /= 2.0f;
          int octet = (int)(x / size) % 2;
          int yi = (int)(y / size) % 2;
          int zi = (int)(z / size) % 2;
          if (yi == 0) octet += 2;
          if (zi == 0) octet += 4;
          k = (k << 3) | (uint64_t)octet;
        }
      }
    }
  } else {
    for (int level = 0; level < levels; ++level) {
      const int o = octets[i * levels + level];
      ok = ok && o >= 0 && o <= 7;
      k = (k << 3) | (uint64_t)(o & 7);
    }
  }
  *key = k;
  return ok;
}

// Octet of a path key at a level (1..levels).
__device__ __forceinline__ int key_octet(uint64_t k, int level, int levels) {
  return (int)(k >> (3 * (levels - level))) & 7;
}

// min(*t, i) into *t; the atomic only where it would change something (a
// value read early is never below the current one).
// HOT: the SM's own cache is asked first, for entries that many points share;
// what it holds was read since the launch began, so it is not below the
// current value either.
template <bool HOT>
__device__ __forceinline__ void propose(uint32_t* t, uint32_t i) {
  if (HOT) {
    uint32_t v;
    asm volatile("ld.global.ca.u32 %0, [%1];" : "=r"(v) : "l"(t));
    if (v <= i) return;
  }
  if (__ldcg(t) > i) atomicMin(t, i);
}

// Whether this lane is the first of its run of lanes with equal s (a run's
// first lane has its smallest point index).
__device__ __forceinline__ bool run_first(uint32_t s) {
  const uint32_t before = __shfl_up_sync(0xFFFFFFFFu, s, 1);
  return (threadIdx.x & 31) == 0 || before != s;
}

// Path keys, the prefix tables of the top levels (reduced in shared memory
// per block first), and for a static build whether the points are in path
// order: own then is the first level each makes, the one after the prefix
// shared with the point before; *unsorted is set where the order, or a point,
// is not so (own is then void: first_kernel sets it).
__global__ void keys_kernel(const float* __restrict__ pts, const int32_t* __restrict__ octets, int64_t n,
                            float basesize, int levels, uint64_t* __restrict__ key, uint8_t* __restrict__ own,
                            uint32_t* __restrict__ dense, unsigned* __restrict__ unsorted, unsigned* __restrict__ err) {
  __shared__ uint32_t sm[kDenseEntries];
  for (int e = threadIdx.x; e < kDenseEntries; e += blockDim.x) sm[e] = kNone;
  __syncthreads();
  const int lane = threadIdx.x & 31, top = levels < kDense ? levels : kDense;
  bool bad = false;
  // a warp takes 32 kKeyGroups consecutive points at a time, so that only the
  // first of them makes the key of the point before it a second time
  constexpr int kSpan = 32 * kKeyGroups;
  const int64_t stride = ((int64_t)gridDim.x * blockDim.x >> 5) * kSpan;
  for (int64_t p0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kSpan; p0 < n; p0 += stride) {
    uint64_t carry = 0;  // key of the point before the group (lane 0)
    if (unsorted && lane == 0 && p0 > 0) bad |= !path_key(pts, octets, p0 - 1, basesize, levels, &carry);
#pragma unroll 1
    for (int g = 0; g < kKeyGroups; ++g) {
      const int64_t i = p0 + 32 * g + lane;
      uint64_t k = kExcluded;
      if (i < n && !path_key(pts, octets, i, basesize, levels, &k)) {
        k = kExcluded;
        atomicOr(err, pts ? kErrBuildPoint : kErrBuildOctet);
      }
      if (i < n) key[i] = k;
      if (unsorted) {
        uint64_t before = __shfl_up_sync(0xFFFFFFFFu, k, 1);
        if (lane == 0) before = carry;
        carry = __shfl_sync(0xFFFFFFFFu, k, 31);
        if (i < n) {
          bad |= k == kExcluded || (i > 0 && k < before);
          own[i] = (uint8_t)(i == 0 ? 1
                             : k == before ? levels + 1
                                           : levels - (63 - __clzll((long long)(k ^ before))) / 3);
        }
      }
      for (int l = 1; l <= top; ++l) {
        const uint32_t s = k == kExcluded ? kNone : (uint32_t)(k >> (3 * (levels - l)));
        const bool first = run_first(s);
        if (s != kNone && first) {
          uint32_t* t = sm + dense_offset(l) + s;
          if (*(volatile uint32_t*)t > (uint32_t)i) atomicMin(t, (uint32_t)i);
        }
      }
    }
  }
  if (bad) *unsorted = 1u;
  __syncthreads();
  for (int e = threadIdx.x; e < kDenseEntries; e += blockDim.x)
    if (sm[e] != kNone) propose<false>(dense + e, sm[e]);
}

// The top levels resolved: the first level each point makes (levels + 1 where
// none yet), its parent's creator, and the first table level proposed.
template <bool HOT>
__global__ void first_kernel(int levels, int64_t from, int64_t n, const uint64_t* __restrict__ key,
                             uint8_t* __restrict__ own, uint32_t* __restrict__ slot, uint32_t* __restrict__ par,
                             const uint32_t* __restrict__ dense, uint32_t* __restrict__ t_prop) {
  const int top = levels < kDense ? levels : kDense;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t b0 = from + (int64_t)blockIdx.x * blockDim.x; b0 < n; b0 += stride) {  // same trip count per block
    const int64_t i = b0 + threadIdx.x;
    const uint64_t k = i < n ? key[i] : kExcluded;
    uint32_t s = kNone;
    if (k != kExcluded) {
      uint32_t c = kNone;  // creator of the level's node; the root's: none
      int o = levels + 1;
      for (int l = 1; l <= top; ++l) {
        const uint32_t w = dense[dense_offset(l) + (uint32_t)(k >> (3 * (levels - l)))];
        if (w == (uint32_t)i && o > levels) {
          o = l;
          par[i] = c;
        }
        c = w;
      }
      own[i] = (uint8_t)o;
      if (t_prop) {
        s = c * 8u + (uint32_t)key_octet(k, top + 1, levels);
        slot[i] = s;
      }
    } else if (i < n) {
      own[i] = (uint8_t)(levels + 1);
    }
    if (t_prop) {
      const bool first = run_first(s);
      if (s != kNone && first) propose<HOT>(t_prop + s, (uint32_t)i);
    }
  }
}

// A point's table slot of a level that it made: its parent's creator is its
// own index below its first level.
__device__ __forceinline__ uint32_t made_slot(uint32_t i, int level, int own, const uint32_t* par, uint64_t k,
                                              int levels) {
  return (own == level ? par[i] : i) * 8u + (uint32_t)key_octet(k, level, levels);
}

// Level l > kDense + 1: resolve level l - 1 (a slot's winner is the creator
// of the group's node; its own slot says its parent's creator), reset the
// entries of level l - 2 (each by its winner, when every point has read it),
// and propose level l.
template <bool HOT>
__global__ void level_kernel(int l, int levels, int64_t from, int64_t n, const uint64_t* __restrict__ key,
                             uint8_t* __restrict__ own, uint32_t* __restrict__ slot, uint32_t* __restrict__ par,
                             const uint32_t* __restrict__ t_res, uint32_t* __restrict__ t_clr,
                             uint32_t* __restrict__ t_prop) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t b0 = from + (int64_t)blockIdx.x * blockDim.x; b0 < n; b0 += stride) {  // same trip count per block
    const int64_t i = b0 + threadIdx.x;
    const uint64_t k = i < n ? key[i] : kExcluded;
    uint32_t s = kNone;
    if (k != kExcluded) {
      const uint32_t so = slot[i];
      const uint32_t c = t_res[so];
      int o = own[i];
      if (c == (uint32_t)i && o > levels) {
        o = l - 1;
        own[i] = (uint8_t)o;
        par[i] = so >> 3;
      }
      if (t_clr && o <= l - 2) t_clr[made_slot((uint32_t)i, l - 2, o, par, k, levels)] = kNone;
      s = c * 8u + (uint32_t)key_octet(k, l, levels);
      slot[i] = s;
    }
    const bool first = run_first(s);
    if (s != kNone && first) propose<HOT>(t_prop + s, (uint32_t)i);
  }
}

// Nodes point i makes (none for one left out: its first level is past the
// last).
__device__ __forceinline__ int32_t made(const uint8_t* own, int64_t i, int64_t n, int levels) {
  return i < n ? max(levels + 1 - (int)own[i], 0) : 0;
}

// Prefix sum, pass 1: nodes made per chunk of PER points a thread. With
// creator tables the deepest level is resolved on the way (t_res; and the
// entries of the level above reset, t_clr), as level_kernel does.
template <int PER>
__global__ void scan_chunks_kernel(uint8_t* __restrict__ own, const uint64_t* __restrict__ key, int64_t n, int levels,
                                   const uint32_t* __restrict__ slot, uint32_t* __restrict__ par,
                                   const uint32_t* __restrict__ t_res, uint32_t* __restrict__ t_clr,
                                   int32_t* __restrict__ blocksum) {
  __shared__ int32_t red[kScanThreads];
  const int64_t b = blockIdx.x;
  int32_t sum = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int64_t i = (b * PER + k) * kScanThreads + threadIdx.x;
    if (i >= n) break;
    int o = own[i];
    if (t_res) {
      const uint64_t kk = key[i];
      if (kk != kExcluded) {
        const uint32_t so = slot[i];
        if (o > levels && t_res[so] == (uint32_t)i) {
          o = levels;
          own[i] = (uint8_t)o;
          par[i] = so >> 3;
        }
        if (t_clr && o <= levels - 1) t_clr[made_slot((uint32_t)i, levels - 1, o, par, kk, levels)] = kNone;
      }
    }
    sum += max(levels + 1 - o, 0);
  }
  red[threadIdx.x] = sum;
  __syncthreads();
  for (int o = kScanThreads / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) blocksum[b] = red[0];
}

// Pass 2 (one block): exclusive scan of the chunk sums in place; the node
// count (with the root) to *total.
__global__ void scan_top_kernel(int32_t* __restrict__ blocksum, int64_t nb, int32_t* __restrict__ total) {
  __shared__ int32_t sh[1024];
  int32_t carry = 1;  // node 0 is the root
  for (int64_t b0 = 0; b0 < nb; b0 += 1024) {
    const int64_t b = b0 + threadIdx.x;
    const int32_t v = b < nb ? blocksum[b] : 0;
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int o = 1; o < 1024; o <<= 1) {
      const int32_t t = threadIdx.x >= o ? sh[threadIdx.x - o] : 0;
      __syncthreads();
      sh[threadIdx.x] += t;
      __syncthreads();
    }
    if (b < nb) blocksum[b] = carry + sh[threadIdx.x] - v;
    const int32_t add = sh[1023];
    __syncthreads();
    carry += add;
  }
  if (threadIdx.x == 0) *total = carry;
}

// Pass 3: each point's first node id; the child blocks and model indices of
// the nodes it makes. A warp takes 32 points at a time; their nodes are one
// run of ids, and its lanes write that run's blocks (two lanes a block) in
// order, whichever point a node belongs to.
template <int PER>
__global__ void spread_kernel(const uint8_t* __restrict__ own, const uint64_t* __restrict__ key, int64_t n, int levels,
                              const int32_t* __restrict__ blocksum, int32_t* __restrict__ base, int64_t first_index,
                              int4* __restrict__ child, int32_t* __restrict__ model, uint32_t* __restrict__ rec) {
  constexpr int kWarps = kScanThreads / 32, kGroups = PER;
  __shared__ int32_t sh[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t p0 = ((int64_t)blockIdx.x * kWarps + warp) * (32 * kGroups);
  int32_t incl[kGroups], sum = 0;
#pragma unroll
  for (int g = 0; g < kGroups; ++g) {
    incl[g] = made(own, p0 + 32 * g + lane, n, levels);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t t = __shfl_up_sync(0xFFFFFFFFu, incl[g], o);
      if (lane >= o) incl[g] += t;
    }
    sum += __shfl_sync(0xFFFFFFFFu, incl[g], 31);
  }
  if (lane == 0) sh[warp] = sum;
  __syncthreads();
  int32_t id = blocksum[blockIdx.x];
  for (int w = 0; w < warp; ++w) id += sh[w];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    // the root: its links and record come later, where it has children
    child[0] = make_int4(0, 0, 0, 0);
    child[1] = make_int4(0, 0, 0, 0);
    model[0] = 0;
    for (int o = 0; o < 8; ++o) {
      rec[2 * o] = 0x00FF00FFu;  // a child without leaves
      rec[2 * o + 1] = 0x000000FFu;
    }
  }
#pragma unroll
  for (int g = 0; g < kGroups; ++g) {
    const int64_t i = p0 + 32 * g + lane;
    const int32_t mine = made(own, i, n, levels);
    const int32_t total = __shfl_sync(0xFFFFFFFFu, incl[g], 31);
    const uint64_t k = mine > 0 ? key[i] : 0ull;
    if (i < n) base[i] = id + incl[g] - mine;
    for (int32_t j0 = 0; j0 < total; j0 += 16) {
      const int32_t j = j0 + (lane >> 1);
      // the point of node j: the first whose nodes end past it
      int q = 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        if (__shfl_sync(0xFFFFFFFFu, incl[g], q + o - 1) <= j) q += o;
      const int32_t end = __shfl_sync(0xFFFFFFFFu, incl[g], q);
      const uint64_t kq = __shfl_sync(0xFFFFFFFFu, k, q);
      if (j < total) {
        const int below = end - 1 - j;  // nodes of the point below this one
        const int32_t node = id + j;
        int4 c = make_int4(0, 0, 0, 0);
        if (below > 0) {
          const int oct = (int)(kq >> (3 * (below - 1))) & 7;
          if ((oct >> 2) == (lane & 1)) {
            c.x = (oct & 3) == 0 ? node + 1 : 0;
            c.y = (oct & 3) == 1 ? node + 1 : 0;
            c.z = (oct & 3) == 2 ? node + 1 : 0;
            c.w = (oct & 3) == 3 ? node + 1 : 0;
          }
        }
        child[2 * (int64_t)node + (lane & 1)] = c;
        if (!(lane & 1)) model[node] = (int32_t)(p0 + 32 * g + q + first_index);
      }
    }
    id += total;
  }
}

// The first node each point makes is linked into its parent, whose id then
// replaces the parent's creator in par. `sorted`: the creator is not known
// yet (par is unset): it is the first point of the parent's prefix. maker
// keeps the creator. t_last: the deepest level's creator table, reset by its
// winners.
__global__ void link_kernel(const uint64_t* __restrict__ key, const uint8_t* __restrict__ own,
                            uint32_t* __restrict__ par, const int32_t* __restrict__ base, int64_t n, int levels,
                            bool sorted, uint32_t* __restrict__ t_last, int32_t* __restrict__ child,
                            uint32_t* __restrict__ maker) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int o = own[i];
    if (o > levels) continue;
    const uint64_t k = key[i];
    if (t_last) t_last[made_slot((uint32_t)i, levels, o, par, k, levels)] = kNone;
    int32_t parent = 0;
    if (o > 1) {
      int64_t p;
      if (sorted) {
        const int sh = 3 * (levels - o + 1);
        const uint64_t first = (k >> sh) << sh;
        // key[lo] < first <= key[hi]; the run starts near i for deep levels
        int64_t hi = i, step = 1, lo = i - 1;
        while (lo >= 0 && key[lo] >= first) {
          hi = lo;
          step *= 2;
          lo = hi - step;
        }
        if (lo < 0) lo = -1;
        while (hi - lo > 1) {
          const int64_t mid = (lo + hi) >> 1;
          if (key[mid] >= first) hi = mid;
          else lo = mid;
        }
        p = hi;
      } else {
        p = par[i];
      }
      parent = base[p] + (o - 1 - own[p]);
      maker[i] = (uint32_t)p;
    }
    par[i] = (uint32_t)parent;
    child[(int64_t)parent * 8 + key_octet(k, o, levels)] = base[i];
  }
}

// Leaf boxes, from every leaf up (see the top). par holds the parent node of
// each point's first node; arrived 4 bits a node, zero.
__global__ void __launch_bounds__(kClimbThreads, 24) climb_kernel(const uint64_t* __restrict__ key, const uint8_t* __restrict__ own,
                             const uint32_t* __restrict__ par, const int32_t* __restrict__ base, int64_t n, int levels,
                             const uint32_t* __restrict__ maker, const int4* __restrict__ child, uint4* box,
                             uint32_t* arrived, uint4* __restrict__ rec) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int o = own[i];
  if (o > levels) return;
  const uint64_t k = key[i];
  int32_t node = base[i] + (levels - o);
  uint32_t p = (uint32_t)i;  // the point whose nodes the climb is among
  CellBox b = {{0u, 0u, 0u}, {0u, 0u, 0u}};
  for (int l = levels - 1; l >= 0; --l) {
    int32_t parent = node - 1;
    if (l + 1 == o) {
      parent = (int32_t)par[p];
      if (l > 0) {
        p = maker[p];
        o = own[p];
      }
    }
    const int sh = levels - 1 - l;
    const int oct = key_octet(k, l + 1, levels);
    int32_t ch[8];
    load_children(child, parent, ch);
    int count = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) count += ch[q] > 0 ? 1 : 0;
    uint2 w[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) w[q] = empty_word();
    CellBox u = no_box();
    if (count == 1) {
      const uint2 r = record_word(b, sh);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q == oct) w[q] = r;
      add_box(u, b, oct, sh);
    } else {
      // the arrival releases this child's box and acquires its siblings'
      __stcg(box + node, pack_box(b));
      const uint32_t at = 4u * ((uint32_t)parent & 7u);
      uint32_t before;
      asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;"
                   : "=r"(before)
                   : "l"(arrived + ((uint32_t)parent >> 3)), "r"(1u << at)
                   : "memory");
      if ((int)((before >> at) & 15u) != count - 1) return;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (ch[q] <= 0) continue;
        const CellBox c = unpack_box(__ldcg(box + ch[q]));
        w[q] = record_word(c, sh);
        add_box(u, c, q, sh);
      }
    }
    b = u;
    store_record(rec, parent, w);
    node = parent;
  }
}

template <typename T>
int grow_buf(T** p, int64_t have, int64_t need, const char* what) {
  if (have >= need && *p) return QBC_OK;
  if (*p) cudaFree(*p);
  *p = nullptr;
  cudaError_t e = cudaMalloc((void**)p, (size_t)std::max<int64_t>(need, 1) * sizeof(T));
  if (e != cudaSuccess) return fail(QBC_E_NOMEM, "tree build scratch (%s, %lld items): %s", what, (long long)need,
                                    cudaGetErrorString(e));
  return QBC_OK;
}

int grid_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  return (int)std::max<int64_t>(1, std::min<int64_t>(b, 65535));
}

}  // namespace

int64_t build_node_bound(int64_t n, int levels) {
  int64_t total = 1, w = 1;
  for (int l = 1; l <= levels; ++l) {
    w = w > ((int64_t)1 << 40) ? w : w * 8;
    total += std::min<int64_t>(n, w);
  }
  return total;
}

void build_release(BuildScratch* s) {
  void* ptrs[] = {s->key, s->slot, s->par, s->base, s->own, s->tab[0], s->tab[1], s->tab[2],
                  s->dense, s->blocksum, s->box, s->arrived};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  *s = BuildScratch();
}

int build_check(int64_t n, int levels) {
  if (n > ((int64_t)1 << 29)) return fail(QBC_E_ARG, "tree build: %lld points exceed 2^29", (long long)n);
  const int64_t nodes = build_node_bound(n, levels);
  if (nodes > INT32_MAX) return fail(QBC_E_ARG, "tree build: up to %lld nodes exceed int32 indices", (long long)nodes);
  return QBC_OK;
}

int build_reserve(BuildScratch* s, int64_t n, int levels) {
  int rc = build_check(n, levels);
  if (rc) return rc;
  const int64_t nodes = build_node_bound(n, levels);
  const int64_t m = std::max<int64_t>(n, 1);
  if (s->points < n || !s->key) {
    s->points = 0;
    ++s->generation;
    if (!rc) rc = grow_buf(&s->key, 0, m, "keys");
    if (!rc) rc = grow_buf(&s->par, 0, m, "parents");
    if (!rc) rc = grow_buf(&s->base, 0, m, "node ids");
    if (!rc) rc = grow_buf(&s->own, 0, m, "levels");
    if (!rc) rc = grow_buf(&s->slot, 0, m, "slots");
    if (rc) return rc;
    s->points = m;
  }
  if (levels > kDense && (s->tab_points < n || !s->tab[0])) {
    s->tab_points = 0;
    ++s->generation;
    for (int t = 0; t < 3 && !rc; ++t) rc = grow_buf(&s->tab[t], 0, 8 * m, "creator tables");
    if (rc) return rc;
    s->tab_points = m;
    s->tables.replaced();  // emptied on the build's stream
  }
  const int64_t nb = scan_chunks_most(n);
  if (s->blocks < nb || !s->blocksum) {
    s->blocks = 0;
    ++s->generation;
    rc = grow_buf(&s->blocksum, 0, std::max<int64_t>(nb, 1), "block sums");
    if (rc) return rc;
    s->blocks = std::max<int64_t>(nb, 1);
  }
  if (s->box_nodes < nodes || !s->box) {
    s->box_nodes = 0;
    ++s->generation;
    rc = grow_buf(&s->box, 0, nodes, "leaf boxes");
    if (!rc) rc = grow_buf(&s->arrived, 0, nodes / 8 + 1, "arrivals");
    if (rc) return rc;
    s->box_nodes = nodes;
  }
  if (!s->dense) {
    ++s->generation;
    rc = grow_buf(&s->dense, 0, kDenseEntries, "prefix tables");
  }
  return rc;
}

namespace {

// Creator table of a level past the prefix tables.
uint32_t* level_table(const BuildScratch* s, int l) { return s->tab[l % 3]; }

// Ids by a prefix sum, once each point's first level (and, unless sorted,
// its parent's creator; with tables, but for the deepest level) is known. The
// node count goes to *total.
void count_nodes(int64_t n, int levels, const BuildScratch* s, bool sorted, int32_t* total, cudaStream_t stream,
                 int64_t* launches) {
  const int64_t nb = scan_chunks(n);
  const bool tables = !sorted && levels > kDense;
  (n <= kScanFew ? scan_chunks_kernel<1> : scan_chunks_kernel<kScanPer>)<<<(unsigned)nb, kScanThreads, 0, stream>>>(
      s->own, s->key, n, levels, s->slot, s->par, tables ? level_table(s, levels) : nullptr,
      tables && levels - 1 > kDense ? level_table(s, levels - 1) : nullptr, s->blocksum);
  scan_top_kernel<<<1, 1024, 0, stream>>>(s->blocksum, nb, total);
  *launches += 2;
}

// Blocks, links and boxes of at most `nodes` nodes. reset: leave the creator
// tables empty for the next build.
void write_tree(int64_t n, int levels, int64_t first_index, const BuildScratch* s, bool sorted, bool reset,
                int64_t nodes, int32_t* child, int32_t* model, uint32_t* rec, cudaStream_t stream,
                int64_t* launches) {
  const int64_t nb = scan_chunks(n);
  (n <= kScanFew ? spread_kernel<1> : spread_kernel<kScanPer>)<<<(unsigned)nb, kScanThreads, 0, stream>>>(
      s->own, s->key, n, levels, s->blocksum, s->base, first_index, reinterpret_cast<int4*>(child), model, rec);
  ++*launches;
  if (n > 0 && levels > 0) {
    const int4* blocks = reinterpret_cast<const int4*>(child);
    uint4* records = reinterpret_cast<uint4*>(rec);
    // (the slots are done: their array takes the parents' creators)
    link_kernel<<<grid_for(n), 256, 0, stream>>>(s->key, s->own, s->par, s->base, n, levels, sorted,
                                                 reset && levels > kDense ? level_table(s, levels) : nullptr, child,
                                                 s->slot);
    ++*launches;
    cudaMemsetAsync(s->arrived, 0, (size_t)(nodes / 8 + 1) * sizeof(uint32_t), stream);
    climb_kernel<<<(unsigned)((n + kClimbThreads - 1) / kClimbThreads), kClimbThreads, 0, stream>>>(
        s->key, s->own, s->par, s->base, n, levels, s->slot, blocks, s->box, s->arrived, records);
    ++*launches;
  }
}

int keys_and_prefixes(const float* d_pts, const int32_t* d_octets, int64_t n, float basesize, int levels,
                      BuildScratch* s, unsigned* unsorted, unsigned* err, cudaStream_t stream, int grid,
                      int64_t* launches) {
  if (levels < 0 || levels > kMaxBuildLevels) return fail(QBC_E_ARG, "tree build: levels %d outside 0..21", levels);
  if (n < 0 || n > s->points) return fail(QBC_E_ARG, "tree build: %lld points beyond the reserved scratch", (long long)n);
  if (cudaMemsetAsync(s->dense, 0xFF, kDenseEntries * sizeof(uint32_t), stream) != cudaSuccess)
    return fail(QBC_E_CUDA, "tree build: reset prefix tables");
  if (n > 0) {
    keys_kernel<<<std::max(1, std::min(grid, grid_for(n))), 256, 0, stream>>>(d_pts, d_octets, n, basesize, levels,
                                                                              s->key, s->own, s->dense, unsorted, err);
    ++*launches;
  }
  return QBC_OK;
}

// After keys_and_prefixes: creators by table (the deepest level's are left to
// count_nodes). any_order: the points may come in any order (see kPilot).
void table_levels(int64_t n, int levels, bool any_order, const BuildScratch* s, cudaStream_t stream, int grid,
                  int64_t* launches) {
  if (n <= 0) return;
  auto level = [&](auto hot, int l, int64_t from, int64_t to) {
    const int g = std::max(1, std::min(grid, grid_for(to - from)));
    if (l == kDense + 1)
      first_kernel<decltype(hot)::value><<<g, 256, 0, stream>>>(levels, from, to, s->key, s->own, s->slot, s->par,
                                                                s->dense,
                                                                levels > kDense ? level_table(s, l) : nullptr);
    else
      level_kernel<decltype(hot)::value><<<g, 256, 0, stream>>>(
          l, levels, from, to, s->key, s->own, s->slot, s->par, level_table(s, l - 1),
          l - 2 > kDense ? level_table(s, l - 2) : nullptr, level_table(s, l));
    ++*launches;
  };
  for (int l = kDense + 1; l <= std::max(levels, kDense + 1); ++l) {
    if (any_order && n >= kPilotMin && l <= kPilotLevel) {
      level(std::false_type{}, l, 0, kPilot);
      level(std::true_type{}, l, kPilot, n);
    } else {
      level(std::false_type{}, l, 0, n);
    }
  }
}

}  // namespace

int build_tree_async(const float* d_pts, const int32_t* d_octets, int64_t n, float basesize, int levels,
                     int64_t first_index, BuildScratch* s, int32_t* child, int32_t* model, uint32_t* rec,
                     int32_t* total, unsigned* err, cudaStream_t stream, int grid, int64_t* launches) {
  const int64_t L0 = *launches;
  int rc = keys_and_prefixes(d_pts, d_octets, n, basesize, levels, s, nullptr, err, stream, grid, launches);
  if (rc) return rc;
  const bool tables = levels > kDense, reset = s->tables.begin(tables);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (reset) {
    if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess) return fail(QBC_E_CUDA, "tree build: capture status");
    for (int t = 0; t < 3; ++t)
      if (cudaMemsetAsync(s->tab[t], 0xFF, (size_t)8 * s->tab_points * sizeof(uint32_t), stream) != cudaSuccess)
        return fail(QBC_E_CUDA, "tree build: reset creator tables");
  }
  table_levels(n, levels, true, s, stream, grid, launches);
  count_nodes(n, levels, s, false, total, stream, launches);
  write_tree(n, levels, first_index, s, false, true, build_node_bound(n, levels), child, model, rec, stream, launches);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    *launches = L0;
    return fail(QBC_E_CUDA, "tree build: %s", cudaGetErrorString(e));
  }
  s->tables.end(tables, reset, capture != cudaStreamCaptureStatusNone);
  return QBC_OK;
}

namespace {

// Device memory of one build, freed when the stream is done with it.
struct Arena {
  cudaStream_t stream;
  std::vector<void*> held;
  explicit Arena(cudaStream_t s) : stream(s) {}
  ~Arena() {
    cudaStreamSynchronize(stream);
    for (void* p : held) cudaFree(p);
  }
  void* take(size_t bytes) {
    void* p = nullptr;
    if (cudaMalloc(&p, std::max<size_t>(bytes, 256)) != cudaSuccess) return nullptr;
    held.push_back(p);
    return p;
  }
};

}  // namespace

int build_tree_static(const float* d_pts, const int32_t* d_octets, int64_t n, float basesize, int levels,
                      int64_t first_index, int32_t* child, int32_t* model, uint32_t* rec, int64_t rec_nodes,
                      int32_t* d_total, int64_t* total, unsigned* flag, unsigned* err, cudaStream_t stream, int grid,
                      int64_t* launches) {
  BuildScratch s;
  Arena arena(stream);
  // per-point state in one allocation, its parts 256-byte aligned
  const int64_t m = std::max<int64_t>(n, 1), nb = scan_chunks(n);
  size_t off = 0;
  auto part = [&](size_t bytes) {
    const size_t at = off;
    off += (bytes + 255) & ~size_t(255);
    return at;
  };
  const size_t key = part(8 * m), par = part(4 * m), base = part(4 * m), own = part(m), slot = part(4 * m),
               sums = part(4 * nb), dense = part(4 * kDenseEntries);
  char* p = static_cast<char*>(arena.take(off));
  if (!p) return fail(QBC_E_NOMEM, "tree build: scratch of %zu bytes", off);
  s.points = n;
  s.key = reinterpret_cast<uint64_t*>(p + key);
  s.par = reinterpret_cast<uint32_t*>(p + par);
  s.base = reinterpret_cast<int32_t*>(p + base);
  s.own = reinterpret_cast<uint8_t*>(p + own);
  s.slot = reinterpret_cast<uint32_t*>(p + slot);
  s.blocksum = reinterpret_cast<int32_t*>(p + sums);
  s.dense = reinterpret_cast<uint32_t*>(p + dense);

  unsigned unsorted = levels > 0 ? 0u : 1u;
  cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(unsigned), stream);
  if (e != cudaSuccess) return fail(QBC_E_CUDA, "tree build: %s", cudaGetErrorString(e));
  int rc = keys_and_prefixes(d_pts, d_octets, n, basesize, levels, &s, levels > 0 ? flag : nullptr, err, stream, grid,
                         launches);
  if (rc) return rc;
  if (levels > 0) {
    e = cudaMemcpyAsync(&unsorted, flag, sizeof(unsigned), cudaMemcpyDeviceToHost, stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return fail(QBC_E_CUDA, "tree build: %s", cudaGetErrorString(e));
  }
  if (unsorted) {
    if (levels > kDense) {
      // the tables lie where the records will be, unless there are too few
      const size_t each = (size_t)32 * m, all = 3 * each;
      char* t = reinterpret_cast<char*>(rec);
      if (all > (size_t)rec_nodes * 64) t = static_cast<char*>(arena.take(all));
      if (!t) return fail(QBC_E_NOMEM, "tree build: creator tables of %zu bytes", all);
      for (int k = 0; k < 3; ++k) s.tab[k] = reinterpret_cast<uint32_t*>(t + k * each);
      e = cudaMemsetAsync(t, 0xFF, all, stream);
      if (e != cudaSuccess) return fail(QBC_E_CUDA, "tree build: %s", cudaGetErrorString(e));
    }
    table_levels(n, levels, false, &s, stream, grid, launches);
  }
  count_nodes(n, levels, &s, !unsorted, d_total, stream, launches);
  int32_t h = 0;
  e = cudaMemcpyAsync(&h, d_total, sizeof(h), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return fail(QBC_E_CUDA, "tree build: %s", cudaGetErrorString(e));
  *total = h;
  // exact boxes and arrival counts past the records, where they fit
  const size_t boxes = (size_t)h * 16, counts = ((size_t)h / 8 + 1) * 4, used = (size_t)h * 64;
  char* t = reinterpret_cast<char*>(rec) + used;
  if (used + boxes + counts > (size_t)rec_nodes * 64) t = static_cast<char*>(arena.take(boxes + counts));
  if (!t) return fail(QBC_E_NOMEM, "tree build: leaf boxes of %zu bytes", boxes + counts);
  s.box = reinterpret_cast<uint4*>(t);
  s.arrived = reinterpret_cast<uint32_t*>(t + boxes);
  write_tree(n, levels, first_index, &s, !unsorted, false, h, child, model, rec, stream, launches);
  e = cudaGetLastError();
  return e == cudaSuccess ? QBC_OK : fail(QBC_E_CUDA, "tree build: %s", cudaGetErrorString(e));
}

namespace {

// ---- octree_remove_point (octree.c:182-218) for a batch of points ----
//
// Per point, the walk of octree_remove_point on the unedited tree: size
// halves from the basecube edge for levels + 1 steps; (int)(c / size) % 2 with
// C truncation and remainder; at level == levels the current node is the
// leaf, reported with its parent and the parent's octet. Points of different
// leaves do not meet (a removal only cuts a parent's link to its leaf), so
// the batch equals sequential calls once duplicates of a leaf are resolved:
// the first in input order removes it, the later ones find the link cut. The
// points claim their leaves in a hash table of at least twice their number
// (leaf << 32 | smallest point index): 0.03 ms for 20K removals, 0.25 by a
// sort of all points with its allocations.
constexpr uint64_t kFree = ~0ull;

__device__ __forceinline__ uint64_t claim_slot(int32_t leaf, uint64_t mask) {
  const uint64_t h = (uint64_t)(uint32_t)leaf * 0x9E3779B97F4A7C15ull;
  return (h ^ (h >> 32)) & mask;
}

__global__ void remove_walk_kernel(const int32_t* __restrict__ child, int64_t n_nodes, const float* __restrict__ pts,
                                   int64_t n, float basesize, int levels, int32_t* __restrict__ leaf,
                                   int32_t* __restrict__ parent, uint8_t* __restrict__ poct,
                                   unsigned long long* claims, uint64_t mask) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float x = pts[3 * i], y = pts[3 * i + 1], z = pts[3 * i + 2];
    float size = basesize;
    int32_t index = 0, lindex = 0, found = -1;
    int loctet = 0;
    for (int level = 0; level < levels + 1; ++level) {
      size /= 2.0f;
      const float qx = x / size, qy = y / size, qz = z / size;
      // a float -> int conversion outside int range is undefined in C: skip
      if (!(fabsf(qx) < 2147483648.0f && fabsf(qy) < 2147483648.0f && fabsf(qz) < 2147483648.0f)) break;
      int octet = (int)qx % 2;
      const int yi = (int)qy % 2, zi = (int)qz % 2;
      if (yi == 0) octet += 2;
      if (zi == 0) octet += 4;
      if (level == levels) {
        found = index;
        break;
      }
      if (octet < 0) break;  // x <= -size: the reference would read oct[-1]
      lindex = index;
      loctet = octet;
      index = child[(int64_t)index * 8 + octet];
      if (index <= 0 || index >= n_nodes) break;  // empty link (or not a node of this tree)
    }
    leaf[i] = found;
    parent[i] = lindex;
    poct[i] = (uint8_t)loctet;
    if (found < 0) continue;
    const unsigned long long mine = ((unsigned long long)(uint32_t)found << 32) | (unsigned long long)i;
    // (at most half the slots are ever taken: a free one comes)
    uint64_t s = claim_slot(found, mask);
    for (uint64_t tries = 0; tries <= mask; ++tries, s = (s + 1) & mask) {
      const unsigned long long was = atomicCAS(claims + s, kFree, mine);
      if (was == kFree) break;
      if ((uint32_t)(was >> 32) == (uint32_t)found) {
        atomicMin(claims + s, mine);
        break;
      }
    }
  }
}

// The first point of each leaf cuts the parent's link and reports the leaf's
// model index and the parent node; the others report -1.
__global__ void remove_apply_kernel(int64_t n, const int32_t* __restrict__ leaf, const int32_t* __restrict__ parent,
                                    const uint8_t* __restrict__ poct, const unsigned long long* __restrict__ claims,
                                    uint64_t mask, int32_t* __restrict__ child, const int32_t* __restrict__ model,
                                    int32_t* __restrict__ modind, int32_t* __restrict__ octind,
                                    unsigned long long* __restrict__ removed) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t b0 = (int64_t)blockIdx.x * blockDim.x; b0 < n; b0 += stride) {  // same trip count per block
    const int64_t i = b0 + threadIdx.x;
    bool first = false;
    if (i < n) {
      const int32_t f = leaf[i];
      if (f >= 0) {
        uint64_t s = claim_slot(f, mask);
        for (uint64_t tries = 0; tries <= mask; ++tries, s = (s + 1) & mask) {
          const unsigned long long k = claims[s];
          if ((uint32_t)(k >> 32) != (uint32_t)f) continue;
          first = (uint32_t)k == (uint32_t)i;
          break;
        }
      }
      if (first) child[(int64_t)parent[i] * 8 + poct[i]] = 0;
      modind[i] = first ? model[f] : -1;
      octind[i] = first ? parent[i] : -1;
    }
    const unsigned all = __ballot_sync(0xFFFFFFFFu, first);
    if ((threadIdx.x & 31) == 0 && all) atomicAdd(removed, (unsigned long long)__popc(all));
  }
}

int64_t claim_slots(int64_t n) {
  int64_t s = 64;
  while (s < 2 * n) s *= 2;
  return s;
}

}  // namespace

size_t remove_scratch(int64_t n) {
  // claims, the count, leaf, parent, octet
  return (size_t)claim_slots(n) * 8 + 8 + (size_t)n * 9;
}

int remove_points(int32_t* child, const int32_t* model, int64_t n_nodes, const float* d_pts, int64_t n,
                  float basesize, int levels, int32_t* d_modind, int32_t* d_octind, void* scratch,
                  unsigned long long** d_removed, cudaStream_t stream, int64_t* launches) {
  if (n >= (int64_t)0xFFFFFFFF) return fail(QBC_E_ARG, "tree remove: %lld points in one call", (long long)n);
  const int64_t slots = claim_slots(n);
  unsigned long long* claims = static_cast<unsigned long long*>(scratch);
  unsigned long long* count = claims + slots;
  int32_t* leaf = reinterpret_cast<int32_t*>(count + 1);
  int32_t* parent = leaf + n;
  uint8_t* poct = reinterpret_cast<uint8_t*>(parent + n);
  cudaError_t e = cudaMemsetAsync(claims, 0xFF, (size_t)slots * 8, stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(count, 0, 8, stream);
  if (e != cudaSuccess) return fail(QBC_E_CUDA, "tree remove: %s", cudaGetErrorString(e));
  remove_walk_kernel<<<grid_for(n), 256, 0, stream>>>(child, n_nodes, d_pts, n, basesize, levels, leaf, parent, poct,
                                                      claims, (uint64_t)slots - 1);
  remove_apply_kernel<<<grid_for(n), 256, 0, stream>>>(n, leaf, parent, poct, claims, (uint64_t)slots - 1, child, model,
                                                       d_modind, d_octind, count);
  *launches += 2;
  *d_removed = count;
  e = cudaGetLastError();
  return e == cudaSuccess ? QBC_OK : fail(QBC_E_CUDA, "tree remove: %s", cudaGetErrorString(e));
}

}  // namespace qbc
