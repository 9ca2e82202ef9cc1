// Internal helpers shared by the translation units of libqbcuda.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "qbcuda.h"
#include "table_state.h"

namespace qbc {

// Record a message for qbc_last_error() and return `code`.
int fail(int code, const char* fmt, ...);
void clear_error();

// True when every cube coordinate of the view's traversal is exactly
// representable, so a child shift can be undone exactly on the way up.
bool cube_shift_exact(const qbc_view& v);

// Device-side input checks that cannot stop a kernel: the kernel records the
// fault in the context's error word and leaves the bad item out; the next
// call that synchronizes with the host (qbc_synchronize, qbc_tree_nodes,
// qbc_download_tree) reports it and clears the word.
enum DeviceError : unsigned {
  kErrBuildPoint = 1u,  // a point to build from was negative, too large or not finite
  kErrBuildOctet = 2u,  // an octet path entry was outside 0..7
  kErrSkinBone = 4u,    // a skinned point named a bone outside the bone set
  kErrMmaTimeout = 8u,  // a bounded wait for the tensor cores gave up (the kernel stopped early)
  kErrRecordOverflow = 16u,  // a split frame's record queue was full (pixels left unwritten)
};

// Scratch of the dynamic tree's GPU build, owned by the context and reused by
// every build: it grows to the largest build seen, so repeated builds of up to that
// size allocate nothing.
struct BuildScratch {
  int64_t points = 0;        // the per-point arrays hold this many points
  int64_t tab_points = 0;    // creator tables hold 8 entries per point for this many
  int64_t blocks = 0;        // prefix-sum block sums
  int64_t box_nodes = 0;     // exact leaf-cell boxes and arrival counts hold this many nodes
  uint64_t* key = nullptr;   // path key, 3 bits per level, root level most significant
  uint32_t* slot = nullptr;  // table slot of the last proposed level, then the creator of par
  uint32_t* par = nullptr;   // creator of the parent of the point's first own node, then the parent's id
  int32_t* base = nullptr;   // id of the point's first own node
  uint8_t* own = nullptr;    // first level whose node the point creates (levels + 1: none)
  uint32_t* tab[3] = {nullptr, nullptr, nullptr};  // creator tables of the deeper levels
  uint32_t* dense = nullptr;  // prefix tables of the top levels
  int32_t* blocksum = nullptr;
  uint4* box = nullptr;      // boxes of nodes with siblings, 6 x 21 bits
  uint32_t* arrived = nullptr;  // children done, 4 bits a node
  TableState tables;         // whether tab's entries are empty
  uint64_t generation = 0;   // raised whenever an array is replaced: captured builds hold their addresses
};

// Nodes a build of n points at `levels` can make: 1 + sum over levels l of
// min(n, 8^l).
int64_t build_node_bound(int64_t n, int levels);

// Whether a build of this size can be numbered.
int build_check(int64_t n, int levels);

// Grow the scratch for n points at `levels` (allocates only when it grows).
int build_reserve(BuildScratch* s, int64_t n, int levels);
void build_release(BuildScratch* s);

// Enqueue on `stream` the node array of inserting n points (d_pts, float3)
// or n octet paths (d_octets, `levels` per point) in order into an empty
// tree (octree_insert_point / octree_insert_path numbering, model indices
// first_index + i), with the leaf-box records (rec, 16 words per node) of
// every node that has children. child (8 int32 per node), model and rec
// must hold build_node_bound(n, levels) nodes; s must have been reserved for
// n points. No allocation and no host synchronisation: the node count is
// written to *total on the device, and a bad point or octet is left out and
// flagged in *err (DeviceError bits).
int build_tree_async(const float* d_pts, const int32_t* d_octets, int64_t n, float basesize, int levels,
                     int64_t first_index, BuildScratch* s, int32_t* child, int32_t* model, uint32_t* rec,
                     int32_t* total, unsigned* err, cudaStream_t stream, int grid, int64_t* launches);

// The same for a build that may wait (two host synchronisations), with
// scratch of its own, freed at the end: 21 bytes a point. It looks whether the
// points are in path order (`flag`: a device word) and then does without the
// creator tables; the tables, and later the exact boxes, lie in the space of
// rec (rec_nodes records) that holds no records yet, or else are allocated.
// The node count goes to *total (d_total: a device word).
int build_tree_static(const float* d_pts, const int32_t* d_octets, int64_t n, float basesize, int levels,
                      int64_t first_index, int32_t* child, int32_t* model, uint32_t* rec, int64_t rec_nodes,
                      int32_t* d_total, int64_t* total, unsigned* flag, unsigned* err, cudaStream_t stream, int grid,
                      int64_t* launches);

// octree_remove_point (octree.c:182-218) of n > 0 points in order, on a device
// tree (child: 8 int32 per node, model: 1 per node): cuts the links in place
// and reports modind / octind per point (-1 where nothing was removed) into
// device arrays; the number removed goes to *d_removed, a device word in
// `scratch` (remove_scratch(n) bytes of device memory, 8-byte aligned).
// Enqueued on `stream`.
size_t remove_scratch(int64_t n);
int remove_points(int32_t* child, const int32_t* model, int64_t n_nodes, const float* d_pts, int64_t n,
                  float basesize, int levels, int32_t* d_modind, int32_t* d_octind, void* scratch,
                  unsigned long long** d_removed, cudaStream_t stream, int64_t* launches);

// Leaf-box records of every node's children (boxes.cu) for the tree `child`
// (8 int32 per node, n nodes) into rec (16 words per node); depth gets the
// tree's depth, or -1 when the array is not a tree the renders can use.
// `scratch`: box_scratch(n) bytes of device memory, 16-byte aligned.
// Synchronizes once, at the end.
size_t box_scratch(int64_t n);
int build_child_boxes(const int32_t* child, int64_t n, uint32_t* rec, void* scratch, cudaStream_t stream, int grid,
                      int* depth, int64_t* launches);

}  // namespace qbc
