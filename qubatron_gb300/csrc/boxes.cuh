// Exact leaf-cell boxes and the record words made of them, shared by the two
// producers of leaf-box records: boxes.cu (uploaded trees) and build.cu
// (trees built on the GPU).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace qbc {

// A box of leaf cells relative to its node: lo x, y, z and hi x, y, z, held
// in memory as 21 bits each. lo > hi: no leaves.
struct CellBox {
  uint32_t lo[3], hi[3];
};
__device__ __forceinline__ CellBox no_box() { return {{0x1FFFFFu, 0x1FFFFFu, 0x1FFFFFu}, {0u, 0u, 0u}}; }

__device__ __forceinline__ uint4 pack_box(const CellBox& b) {
  const uint64_t l = (uint64_t)b.lo[0] | ((uint64_t)b.lo[1] << 21) | ((uint64_t)b.lo[2] << 42);
  const uint64_t h = (uint64_t)b.hi[0] | ((uint64_t)b.hi[1] << 21) | ((uint64_t)b.hi[2] << 42);
  return make_uint4((uint32_t)l, (uint32_t)(l >> 32), (uint32_t)h, (uint32_t)(h >> 32));
}
__device__ __forceinline__ CellBox unpack_box(uint4 v) {
  const uint64_t l = (uint64_t)v.x | ((uint64_t)v.y << 32), h = (uint64_t)v.z | ((uint64_t)v.w << 32);
  CellBox b;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    b.lo[a] = (uint32_t)(l >> (21 * a)) & 0x1FFFFFu;
    b.hi[a] = (uint32_t)(h >> (21 * a)) & 0x1FFFFFu;
  }
  return b;
}

// Box b of child q, whose edge has 2^sh leaf cells, added to its node's u.
__device__ __forceinline__ void add_box(CellBox& u, const CellBox& b, int q, int sh) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const uint32_t off = ((q >> a) & 1) ? 1u << sh : 0u;
    u.lo[a] = min(u.lo[a], b.lo[a] + off);
    u.hi[a] = max(u.hi[a], b.hi[a] + off);
  }
}

// Record word of a child of 2^sh leaf cells an edge with box b: [lo, hi + 1)
// in 1/256 of the edge, rounded outward.
__device__ __forceinline__ uint2 record_word(const CellBox& b, int sh) {
  uint32_t q[6];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const uint32_t lo = b.lo[a], hi1 = b.hi[a] + 1u;
    q[2 * a] = sh >= 8 ? lo >> (sh - 8) : lo << (8 - sh);
    q[2 * a + 1] = (sh >= 8 ? (hi1 + (1u << (sh - 8)) - 1u) >> (sh - 8) : hi1 << (8 - sh)) - 1u;
  }
  return make_uint2(q[0] | (q[1] << 8) | (q[2] << 16) | (q[3] << 24), q[4] | (q[5] << 8));
}
// ... and of a child without leaves, or of none.
__device__ __forceinline__ uint2 empty_word() { return make_uint2(0x00FF00FFu, 0x000000FFu); }

// A node's child block, and its record, by 32-byte accesses (whole sectors).
__device__ __forceinline__ void load_children(const int4* child, int32_t node, int32_t (&ch)[8]) {
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(ch[0]), "=r"(ch[1]), "=r"(ch[2]), "=r"(ch[3]), "=r"(ch[4]), "=r"(ch[5]), "=r"(ch[6]), "=r"(ch[7])
               : "l"(child + 2 * (int64_t)node));
}

__device__ __forceinline__ void store_record(uint4* rec, int32_t node, const uint2 (&w)[8]) {
#pragma unroll
  for (int q = 0; q < 2; ++q)
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(rec + (int64_t)node * 4 + 2 * q),
                 "r"(w[4 * q].x), "r"(w[4 * q].y), "r"(w[4 * q + 1].x), "r"(w[4 * q + 1].y), "r"(w[4 * q + 2].x),
                 "r"(w[4 * q + 2].y), "r"(w[4 * q + 3].x), "r"(w[4 * q + 3].y)
                 : "memory");
}

}  // namespace qbc
