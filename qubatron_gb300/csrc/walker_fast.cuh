// The walk of walker.cuh with the subnode test in parametric form, for exact
// basecubes whose trees all have usable leaf boxes. Same leaves, entry points
// and visit counts, bit for bit.
//
// The shader orders a cube's candidates by computing the points where the ray
// meets the three bisecting planes and comparing their coordinates with the
// cube. For almost every cube those comparisons follow from the ray's t at the
// planes alone: the octet of the entry point is given by the planes crossed
// before the entry t, and every plane crossed before the exit t starts the
// next octet. step() works on the t values, and first checks that no two
// of the t values it compares are closer than the rounding errors, its own and
// the shader's, could bridge (`guard`). Where two are, list_exact() does the
// shader's arithmetic from the exact entry point, for this cube and the
// subtree below it (0.05-0.2 % of the visits).
//
// What bounds it: instruction issue (70 % of the cycles) and the ALU pipe (69 %
// busy; DRAM 2 % of its rate): a 1920x1080 view of a 5M-point room takes 2.69G
// warp instructions for 201M node visits. A step has no divergent branch but
// the ambiguous one: all four list entries are read and tested at once, the
// two bounds of an axis in one packed FMA, the octet bits are carried in the
// t values' low bits, and a descent reads its own list back from the stack as
// a pop does (branches around the reads and the descent cost 8 %). Against
// walker.cuh's walk in the same kernel, 16 x 1080p of a 20M-point room take
// 34.0 instead of 57.0 ms; 2M random rays in a 2M-point room 1.52 instead of
// 2.57. 6 blocks of 128 threads per SM (80 registers); 7 (18 bytes spilled)
// measured the same, 8 spill 94 bytes and take 1.6x. Prefetching the next
// node's record cost 3 % of a frame and half as much again of random rays.
//
// Path. The corner of the current cube is held per axis as the float 1 + path
// bits (bit 22 - k for level k), so fma(X, S, -S) is the exact coordinate, a
// pop masks mantissa bits and a descent sets one.
//
// Stack, [level][word][thread] as in walker.cuh:
//   word 0  4 entries of 5 bits (octet | source << 3; source 0, 1, 2 the
//           x, y, z bisecting plane, 3 the cube's own entry point), bits
//           20-23 the entries still to take for the static tree, 24-27 for
//           the dynamic tree, 28-29 the entry last taken, 30 set when
//           list_exact() made the list;
//   word 1, 2  the level's static and dynamic node index.
#pragma once

#include "walker.cuh"

namespace qbc {

// 0x4B0000bb-style byte pick: bytes of a (0-3) and b (4-7); a nibble with its
// top bit set replicates the picked byte's sign bit.
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

// A ray at a cube: what the out-of-line parts of the walk take.
struct Spot {
  float3 p, d, inv;
  float s;  // basecube edge
  uint32_t X, Y, Z;
  uint32_t mode;
  int level;
};

// Coordinates of a path value: exact, since X * S / 2^L is representable.
__device__ __forceinline__ float path_up(uint32_t f, float s) { return __fmaf_rn(__uint_as_float(f), s, -s); }
__device__ __forceinline__ float path_down(uint32_t f, float s) { return __fmaf_rn(-__uint_as_float(f), s, s + s); }

// Point where the ray meets the plane c of an axis, by the shader's
// operations.
__device__ __forceinline__ float4 axis_plane_hit(const Spot& r, int axis, float c) {
  const float pa = axis == 0 ? r.p.x : (axis == 1 ? r.p.y : r.p.z);
  const float da = axis == 0 ? r.d.x : (axis == 1 ? r.d.y : r.d.z);
  const float ya = axis == 0 ? r.inv.x : (axis == 1 ? r.inv.y : r.inv.z);
  const float w = (r.mode & 1u) ? div_by_recip(c - pa, da, ya) : (c - pa) / (da == 0.0f ? 1.0f : da);
  return make_float4(axis == 0 ? c : r.p.x + r.d.x * w, axis == 1 ? c : r.p.y + r.d.y * w,
                     axis == 2 ? c : r.p.z + r.d.z * w, w);
}

// Basecube entry point (octree_fsh.c:157-211): false for a discard.
__device__ __forceinline__ bool base_entry(float3 p, float3 d, float s, float4& h0) {
  Walker<true, false> w;
  w.p = p;
  w.d = d;
  return w.entry(make_float4(0.0f, s, s, s), h0);
}

// Exact entry point of a cube: the plane that the nearest level above entered
// through one of its own planes, or the basecube's entry. `words` stack words
// a level.
static __device__ __forceinline__ float4 cube_entry(const Spot r, const uint32_t* stack, int stride, int words) {
  for (int l = r.level - 1; l >= 0; --l) {
    const uint32_t pk = stack[words * l * stride];
    const int src = (int)((pk >> (5 * ((pk >> 28) & 3u))) >> 3) & 3;
    if (src != 3) {
      const uint32_t bit = 0x00400000u >> l, keep = 0xFFFFFFFFu << (23 - l);
      const uint32_t f = ((src == 0 ? r.X : (src == 1 ? r.Y : r.Z)) & keep) | bit;
      return axis_plane_hit(r, src, src == 0 ? path_up(f, r.s) : path_down(f, r.s));
    }
  }
  float4 h;
  base_entry(r.p, r.d, r.s, h);
  return h;
}

// The shader's candidates of a cube (octree_fsh.c:251-329) before its
// occupancy test, from its arithmetic: the packed entries, their number in
// bits 20-22. See Walker::step for the forms used.
static __device__ __forceinline__ uint32_t list_exact(const Spot r, const uint32_t* stack, int stride, int words) {
  const float w = r.s * __int_as_float((127 - r.level) << 23);
  const float4 cube = make_float4(path_up(r.X, r.s), path_down(r.Y, r.s), path_down(r.Z, r.s), w);
  const float4 e = cube_entry(r, stack, stride, words);
  const float4 cb = brb_of(cube);
  const float3 hl = hlf_of(cube);
  const float4 hz = axis_plane_hit(r, 2, hl.z), hx = axis_plane_hit(r, 0, hl.x), hy = axis_plane_hit(r, 1, hl.y);
  const bool vz = (r.d.z != 0.0f) & (hz.w > 0.0f) & in_zface(hz, cube, cb);
  const bool vx = (r.d.x != 0.0f) & (hx.w > 0.0f) & in_xface(hx, cube, cb);
  const bool vy = (r.d.y != 0.0f) & (hy.w > 0.0f) & in_yface(hy, cube, cb);
  const float kInf = __int_as_float(0x7f800000);
  // code: octet | source << 3 | the octet bit the pair fix-up flips << 5
  float t[4] = {e.w, vz ? hz.w : kInf, vx ? hx.w : kInf, vy ? hy.w : kInf};
  uint32_t c[4];
  c[0] = (e.x > hl.x ? 1u : 0u) | (e.y < hl.y ? 2u : 0u) | (e.z < hl.z ? 4u : 0u) | (3u << 3) |
         (e.x == hl.x ? 1u << 5 : (e.y == hl.y ? 2u << 5 : (e.z == hl.z ? 4u << 5 : 0u)));
  c[1] = (hz.x > hl.x ? 1u : 0u) | (hz.y < hl.y ? 2u : 0u) | (2u << 3) |
         (hz.x == hl.x ? 1u << 5 : (hz.y == hl.y ? 2u << 5 : 4u << 5));
  c[2] = (hx.y < hl.y ? 2u : 0u) | (hx.z < hl.z ? 4u : 0u) | (1u << 5);
  c[3] = (hy.x > hl.x ? 1u : 0u) | (hy.z < hl.z ? 4u : 0u) | (1u << 3) | (hy.x == hl.x ? 1u << 5 : 2u << 5);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = i + 1; j < 4; ++j)
      if (t[j] < t[i]) {
        const float tt = t[i];
        t[i] = t[j];
        t[j] = tt;
        const uint32_t cc = c[i];
        c[i] = c[j];
        c[j] = cc;
      }
  const int n = 1 + (int)vz + (int)vx + (int)vy;
  uint32_t pk = 0u, pre = 8u;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t o = c[i] & 7u;
    if (o == pre) o ^= c[i] >> 5;
    pre = o;
    if (i < n) pk |= (o | (c[i] & 24u)) << (5 * i);
  }
  return pk | (uint32_t)n << 20;
}

// Instrumented renders: the box words the filter reads at a node, counted as
// Walker::step counts them (entries whose child exists).
__device__ __forceinline__ uint32_t words_read(const int32_t* child, int32_t node, uint32_t pk, int n) {
  uint32_t nw = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (i < n) nw += __ldg(child + 8 * (size_t)(uint32_t)node + ((pk >> (5 * i)) & 7u)) > 0 ? 1u : 0u;
  return nw;
}

// Pairs of floats for the packed operations: f.x * u.x + c.x, f.y * u.y + c.y
// (held as 64-bit registers: a pair used more than once is built once).
using f2 = unsigned long long;
__device__ __forceinline__ f2 pair(float x, float y) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpair(f2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// INSTR: instrumented walks (a visits output, render statistics) use
// child_box_hit's own operations, so that their visit counts are those of the
// walk in walker.cuh. The others use a cheaper box test within the same
// margin, and descend into a tree only where its own box is met. The leaves
// are the same.
template <bool DYN, bool INSTR, bool PROP = false>
struct FastWalker {
  float3 p;      // ray origin
  float3 inv;    // RN(1 / d) per component of the direction (0 for a zero component)
  // bit 0 plane hits may divide by reciprocal (div_by_recip); bit 1 the ray
  // allows boxes and the parametric test; bit 3 it leaves the dynamic tree
  // alone; bits 4-6 the octet a ray from before all three planes starts in
  uint32_t mode;
  uint32_t selx, sely, selz;  // prmt selectors of the near bounds in a box word
  float guard;                // 1.25 * 2^-24 * S * max |inv|
  uint32_t X, Y, Z;           // bits of 1 + path per axis
  uint32_t more;              // bit L set when level L's list has entries to take
  int level;
  int32_t ns, nd;
  bool slow;                  // this cube lies below an ambiguous one (or the ray allows no boxes)
  bool oob;
  uint32_t vis_s, vis_d;
  uint32_t words;  // INSTR: leaf-box words the lane's walks read (sc.box_words set)
  // proposal test (PROP only): above tdepth the walk takes only the first
  // entry towards the cell of path `target` (3 bits per level, root first);
  // no entries are left there, so pops stop at tdepth
  uint32_t target;
  int tdepth;

  static constexpr int kWords = DYN ? 3 : 2;
  static constexpr uint32_t kEmptyBox = 0x00FF00FFu;  // word x of a child without leaves
  // selectors: bound byte b of axis a becomes a float's bytes by prmt with
  // the octet's bit of the axis (256 units) and an exponent byte; INSTR
  // 2^23 + units, else 2^15 + units with the bound in byte 1
  static constexpr uint32_t kBound = INSTR ? 1u : 16u;  // the other bound of the axis: ^ kBound
  static __device__ __forceinline__ uint32_t selector(uint32_t axis, uint32_t b) {
    return INSTR ? 0x7F40u | (axis << 4) | b : 0x740Fu | (axis << 8) | (b << 4);
  }

  __device__ __forceinline__ uint32_t& slot(const Stack& st, int l, int k) const {
    return st.base[(kWords * l + k) * st.stride];
  }

  __device__ __forceinline__ Spot spot(float3 d, float s) const { return {p, d, inv, s, X, Y, Z, mode, level}; }

  // Start a ray: the basecube entry. Returns kDiscard or kRunning.
  __device__ __forceinline__ int start(float4 bc, float3 rp, float3 d, const DevScene& sc, int maxlevel) {
    (void)maxlevel;  // the launch's trees all have boxes down to it
    p = rp;
    X = Y = Z = 0x3F800000u;
    more = 0u;
    level = 0;
    ns = 0;
    nd = 0;
    oob = false;
    vis_s = 0;
    vis_d = 0;
    target = 0u;
    tdepth = 0;
    const float s = bc.w;
    const bool fdiv = recip_div_ok(p, d, s);
    const bool geo = box_ray_ok(p, d, s, fdiv);
    inv = make_float3(d.x == 0.0f ? 0.0f : __frcp_rn(d.x), d.y == 0.0f ? 0.0f : __frcp_rn(d.y),
                      d.z == 0.0f ? 0.0f : __frcp_rn(d.z));
    mode = (fdiv ? 1u : 0u) | (geo ? 2u : 0u) | (d.x < 0.0f ? 16u : 0u) | (d.y > 0.0f ? 32u : 0u) |
           (d.z > 0.0f ? 64u : 0u);
    if (DYN && geo && !root_box_near(sc.tree[1], bc, p, inv)) mode |= 8u;
    // bytes of a box word: xlo xhi ylo yhi, then zlo zhi; y and z count
    // against their axes
    selx = selector(0u, inv.x > 0.0f ? 0u : 1u);
    sely = selector(1u, inv.y > 0.0f ? 3u : 2u);
    selz = selector(2u, inv.z > 0.0f ? 1u : 0u);
    const float mi = fmaxf(fabsf(inv.x), fmaxf(fabsf(inv.y), fabsf(inv.z)));
    guard = 7.4505806e-08f * (s * mi);  // 1.25 * 2^-24
    // The basecube's faces by t: where no two of the t values that decide are
    // closer than the errors, the shader's face tests pass for the entry and
    // the exit face alone, or (a miss, or the cube behind the origin) it
    // discards. Else its own arithmetic decides: six face hits, each with a
    // division (for nearly every ray they were the start's largest part).
    const float x0 = (0.0f - p.x) * inv.x, x1 = (s - p.x) * inv.x;
    const float y0 = (0.0f - p.y) * inv.y, y1 = (s - p.y) * inv.y;
    const float z0 = (0.0f - p.z) * inv.z, z1 = (s - p.z) * inv.z;
    const float nx = fminf(x0, x1), ny = fminf(y0, y1), nz = fminf(z0, z1);
    const float fx = fmaxf(x0, x1), fy = fmaxf(y0, y1), fz = fmaxf(z0, z1);
    const float t0 = fmaxf(fmaxf(nx, ny), nz), t1 = fminf(fminf(fx, fy), fz);
    const float n2 = fmaxf(fminf(nx, ny), fminf(fmaxf(nx, ny), nz));  // the second near and far t
    const float f2 = fminf(fmaxf(fx, fy), fmaxf(fminf(fx, fy), fz));
    const float g = __fmaf_rn(fmaxf(fabsf(t0), fabsf(t1)), kRelGuard, guard);
    if (geo && (t0 > t1 + g || t1 < -g)) return kDiscard;
    slow = !geo;
    if (!(geo && t1 > t0 + g && t1 > g && t0 - n2 > g && f2 - t1 > g && fabsf(t0) > g)) {
      float4 h0;
      if (!base_entry(p, d, s, h0)) return kDiscard;
      // the walk takes the largest near t for the entry t: at a basecube edge
      // the shader may have picked another face
      slow |= !(fabsf(h0.w - fmaxf(t0, 0.0f)) <= g);
    }
    return kRunning;
  }

  static constexpr float kRelGuard = 2.8610229e-06f;  // 48 * 2^-24

  // After start(): whether a two-tree walk of this ray reads the dynamic
  // tree, i.e. FastWalker<true>::start would not give it mode bit 3.
  __device__ __forceinline__ bool walks_dynamic(const DevScene& sc, float4 bc, int maxlevel) const {
    const DevTree& t = sc.tree[1];
    if (!(mode & 2u) || t.cbox == nullptr || maxlevel < t.box_depth) return true;
    return root_box_near_call(t.child, t.cbox, t.box_depth, t.n, bc, p, inv);
  }

  // One step: the list of the current (freshly entered) cube, then the
  // nearest level with entries to take and the descent into its next one.
  // dir() gives the ray's direction. Returns kRunning, kLeaf or kMiss.
  template <class Dir>
  __device__ __forceinline__ int step(const DevScene& sc, int maxlevel, float4 bc, const Stack& st, Dir dir) {
    const float s = bc.w;
    // trees with a node at this cube (none at maxlevel: see the end)
    const bool dl = DYN && !(mode & 8u);
    const bool has_s = DYN ? ns > 0 || level == 0 : level < maxlevel;
    const bool has_d = dl && (nd > 0 || level == 0);
    if (INSTR) {
      if (has_s) ++vis_s;
      if (has_d) ++vis_d;
    }

    // ---- the ray's t at the cube's planes (box_frame's terms) ----
    const bool geo = (mode & 2u) != 0u;
    const float lv2 = __int_as_float((127 - level) << 23);  // 2^-level
    const float ax = (path_up(X, s) - p.x) * inv.x;
    const float ay = (path_down(Y, s) - p.y) * inv.y;
    const float az = (path_down(Z, s) - p.z) * inv.z;
    const float unit = (s * 0.001953125f) * lv2;  // 1/512 of the edge
    const float ux = unit * inv.x, uy = -(unit * inv.y), uz = -(unit * inv.z);

    const float kInf = __int_as_float(0x7f800000);
    uint32_t o[4], pk;
    bool v[4];
    bool exact;
    v[0] = true;
    {
      const float tx = __fmaf_rn(256.0f, ux, ax), ty = __fmaf_rn(256.0f, uy, ay), tz = __fmaf_rn(256.0f, uz, az);
      const float t0 = fmaxf(fmaxf(fmaxf(__fmaf_rn(-256.0f, fabsf(ux), tx), __fmaf_rn(-256.0f, fabsf(uy), ty)),
                                   __fmaf_rn(-256.0f, fabsf(uz), tz)),
                             0.0f);
      const float t1 = fminf(fminf(__fmaf_rn(256.0f, fabsf(ux), tx), __fmaf_rn(256.0f, fabsf(uy), ty)),
                             __fmaf_rn(256.0f, fabsf(uz), tz));
      // no two of the compared values closer than the errors
      const float ga = fminf(fminf(fabsf(tx - t0), fabsf(ty - t0)), fabsf(tz - t0));
      const float gb = fminf(fminf(fabsf(tx - t1), fabsf(ty - t1)), fabsf(tz - t1));
      const float gc = fminf(fminf(fabsf(tx - ty), fabsf(ty - tz)), fabsf(tz - tx));
      const float lim = __fmaf_rn(t1, kRelGuard, __fmaf_rn(8.0f * lv2, guard, guard));
      exact = slow | !(fminf(fminf(ga, gb), gc) > lim);
      // planes not yet crossed at the entry, in order of t; those past t1 are
      // crossed outside. A t's three lowest bits hold its plane's octet bit.
      const bool bx = tx < t0, by = ty < t0, bz = tz < t0;
      const float kx = bx ? kInf : __uint_as_float((__float_as_uint(tx) & ~7u) | 1u);
      const float ky = by ? kInf : __uint_as_float((__float_as_uint(ty) & ~7u) | 2u);
      const float kz = bz ? kInf : __uint_as_float((__float_as_uint(tz) & ~7u) | 4u);
      const float m1 = fminf(kx, ky), m2 = fmaxf(kx, ky);
      const float k1 = fminf(m1, kz), m3 = fmaxf(m1, kz);
      const float k2 = fminf(m2, m3), k3 = fmaxf(m2, m3);
      const uint32_t b1 = __float_as_uint(k1), b2 = __float_as_uint(k2), b3 = __float_as_uint(k3);
      o[0] = ((bx ? 1u : 0u) | (by ? 2u : 0u) | (bz ? 4u : 0u)) ^ ((mode >> 4) & 7u);
      o[1] = o[0] ^ (b1 & 7u);
      o[2] = o[1] ^ (b2 & 7u);
      o[3] = o[2] ^ (b3 & 7u);
      v[1] = k1 < t1;
      v[2] = k2 < t1;
      v[3] = k3 < t1;
      // (octet bits 1, 2, 4 to sources 0, 1, 2)
      pk = (((o[3] | ((b3 << 2) & 24u)) * 32u + (o[2] | ((b2 << 2) & 24u))) * 32u + (o[1] | ((b1 << 2) & 24u))) * 32u +
           (o[0] + 24u);
    }
    if (__builtin_expect(exact, 0)) {
      pk = list_exact(spot(dir(), s), st.base, st.stride, kWords);
      const int n = (int)(pk >> 20);
      pk &= 0xFFFFFu;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        o[i] = (pk >> (5 * i)) & 7u;
        v[i] = i < n;
      }
    }

    // ---- leaf boxes of the listed children ----
    f2 cx, cy, cz;  // near and far terms of a bound
    if (INSTR) {
      // child_box_hit's a0 and a1, the near one first
      const float m = s * 6.1035156e-05f;  // 2^-14 S
      const float mx = fabsf(m * inv.x), my = fabsf(m * inv.y), mz = fabsf(m * inv.z);
      cx = pair(ax - mx, ax + mx);
      cy = pair(ay - my, ay + my);
      cz = pair(az - mz, az + mz);
    } else {
      // a bound's float is 2^15 + units, a high bound's cell ends one unit
      // later (half a unit either way from the middle), and 2^-14 S is
      // 2^(level - 5) units; 0.01 unit covers the rounding of these terms
      const float k = 0.51f + __int_as_float((127 - 5 + level) << 23);
      const float bx = __fmaf_rn(ux, -32767.5f, ax), by = __fmaf_rn(uy, -32767.5f, ay),
                  bz = __fmaf_rn(uz, -32767.5f, az);
      cx = pair(__fmaf_rn(fabsf(ux), -k, bx), __fmaf_rn(fabsf(ux), k, bx));
      cy = pair(__fmaf_rn(fabsf(uy), -k, by), __fmaf_rn(fabsf(uy), k, by));
      cz = pair(__fmaf_rn(fabsf(uz), -k, bz), __fmaf_rn(fabsf(uz), k, bz));
    }
    const f2 u2x = pair(ux, ux), u2y = pair(uy, uy), u2z = pair(uz, uz);
    auto meets = [&](uint2 r, uint32_t oct) {
      // bytes 0, 1, 2: the octet's x, y, z bit; byte 3: the exponent
      const uint32_t b = ((oct * 0x4081u) & 0x00010101u) | (INSTR ? 0x4B000000u : 0x47000000u);
      auto bounds = [&](uint32_t w, uint32_t sel) {
        return pair(__uint_as_float(prmt(w, b, sel)), __uint_as_float(prmt(w, b, sel ^ kBound)));
      };
      f2 qx = bounds(r.x, selx), qy = bounds(r.x, sely), qz = bounds(r.y, selz);
      if (INSTR) {
        // a high bound (an odd byte): one unit more
        auto off = [](uint32_t sel) {
          const float k = (sel & 1u) ? -8388607.0f : -8388608.0f;
          return pair(k, -16777215.0f - k);
        };
        qx = add2(qx, off(selx));
        qy = add2(qy, off(sely));
        qz = add2(qz, off(selz));
      }
      const float2 tx = unpair(fma2(qx, u2x, cx)), ty = unpair(fma2(qy, u2y, cy)), tz = unpair(fma2(qz, u2z, cz));
      const float tn = fmaxf(fmaxf(tx.x, ty.x), tz.x), tf = fminf(fminf(tx.y, ty.y), tz.y);
      // (a box behind the origin: listed cubes are not, so INSTR alone asks)
      return (tn <= tf) & (!INSTR | (tf >= 0.0f));
    };
    // entries of a tree's node: the children with leaves (an empty child's
    // record says so) whose box the ray meets (the deepest level's children
    // are leaf cells, their boxes whole: every listed entry meets them). All
    // four are tested, listed or not: the lanes of a warp nearly always list
    // four between them. Only the listed are read: reading all four cost
    // incoherent rays the record's other sector (4M rays 4.34 ms, 4.02 so).
    auto filter = [&](const DevTree& t, int32_t node) {
      const uint2* rec = reinterpret_cast<const uint2*>(t.cbox) + (size_t)(uint32_t)node * 8;
      uint2 r[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] = v[i] ? __ldg(rec + o[i]) : make_uint2(kEmptyBox, 0u);
      uint32_t keep = 0u;
#pragma unroll
      for (int i = 0; i < 4; ++i) keep |= ((r[i].x != kEmptyBox) & meets(r[i], o[i])) ? 1u << i : 0u;
      if (__builtin_expect(!geo, 0)) {  // the shader's own test (octree_fsh.c:313-317)
        const int32_t* c = reinterpret_cast<const int32_t*>(t.child) + 8 * (size_t)(uint32_t)node;
        keep = 0u;
        for (int i = 0; i < 4; ++i)
          if (v[i] && __ldg(c + ((pk >> (5 * i)) & 7u)) > 0) keep |= 1u << i;
      }
      return level < t.box_depth ? keep : 0u;
    };
    uint32_t ks = 0u, kd = 0u;
    if (!DYN) ks = filter(sc.tree[0], ns);
    else if (has_s) ks = filter(sc.tree[0], ns);
    if (DYN && has_d) kd = filter(sc.tree[1], nd);
    if (INSTR && sc.box_words) {
      const int n = 1 + (int)v[1] + (int)v[2] + (int)v[3];
      if (geo && has_s && level + 1 < sc.tree[0].box_depth)
        words += words_read(reinterpret_cast<const int32_t*>(sc.tree[0].child), ns, pk, n);
      if (DYN && geo && has_d && level + 1 < sc.tree[1].box_depth)
        words += words_read(reinterpret_cast<const int32_t*>(sc.tree[1].child), nd, pk, n);
    }
    // ---- take the next entry (octree_fsh.c:334-375) ----
    // The list goes to the stack and the nearest level with entries left is
    // read back, also where that is this one: descending and popping lanes
    // follow one sequence without a branch.
    if (PROP && level < tdepth) {
      const uint32_t want = target >> (3 * (tdepth - 1 - level));
      uint32_t to = 0u;
#pragma unroll
      for (int i = 0; i < 4; ++i) to |= (((pk >> (5 * i)) ^ want) & 7u) == 0u ? 1u << i : 0u;
      to &= ks | kd;
      to &= 0u - to;  // the first
      ks &= to;
      kd &= to;
    }
    const uint32_t all = DYN ? ks | kd : ks;
    if (all) {
      slot(st, level, 0) = pk | (ks << 20) | (DYN ? kd << 24 : 0u) | (exact ? 1u << 30 : 0u);
      slot(st, level, 1) = (uint32_t)ns;
      if (DYN) slot(st, level, 2) = (uint32_t)nd;
      more |= 1u << level;
    }
    if (more == 0u) return kMiss;
    const int lv = 31 - __clz((int)more);
    pk = slot(st, lv, 0);
    const int32_t node = (int32_t)slot(st, lv, 1);
    const uint32_t left = (DYN ? (pk >> 20) | (pk >> 24) : pk >> 20) & 15u;
    const int i = __ffs((int)left) - 1;
    const int oct = (int)((pk >> (5 * i)) & 7u);
    int32_t cs = 0, cd = 0;
    bool ok;
    if (DYN) {
      const int32_t node_d = (int32_t)slot(st, lv, 2);
      const bool hs = (pk >> (20 + i)) & 1u, hd = (pk >> (24 + i)) & 1u;
      if ((INSTR || hs) && (node > 0 || lv == 0))
        cs = __ldg(reinterpret_cast<const int32_t*>(sc.tree[0].child) + 8 * (size_t)(uint32_t)node + oct);
      if (dl && (INSTR || hd) && (node_d > 0 || lv == 0))
        cd = __ldg(reinterpret_cast<const int32_t*>(sc.tree[1].child) + 8 * (size_t)(uint32_t)node_d + oct);
      ok = (hs && cs > 0) || (hd && cd > 0);
    } else {
      cs = __ldg(reinterpret_cast<const int32_t*>(sc.tree[0].child) + 8 * (size_t)(uint32_t)node + oct);
      ok = cs > 0;
    }
    slot(st, lv, 0) = (pk & ~((3u << 28) | ((DYN ? 0x01100000u : 0x00100000u) << i))) | ((uint32_t)i << 28);
    if ((left & (left - 1u)) == 0u) more &= ~(1u << lv);
    const uint32_t keep = 0xFFFFFFFFu << (23 - lv), bit = 0x00400000u >> lv;
    X = (X & keep) | ((oct & 1) ? bit : 0u);
    Y = (Y & keep) | ((oct & 2) ? bit : 0u);
    Z = (Z & keep) | ((oct & 4) ? bit : 0u);
    slow = (pk >> 30) != 0u;
    // a removed node's link is cut while its box stays: the lane goes on from
    // the root's record at maxlevel, at and below every tree's depth, where
    // the filter lists nothing, so its next step takes another entry
    level = ok ? lv + 1 : maxlevel;
    ns = ok ? cs : 0;
    nd = ok ? cd : 0;
    return ok & (level == maxlevel) ? kLeaf : kRunning;
  }

  // Entry point of the leaf cell; call after step() returned kLeaf.
  __device__ __forceinline__ float4 leaf_point(const Stack& st, float4 bc, float3 d) const {
    return cube_entry(spot(d, bc.w), st.base, st.stride, kWords);
  }

  // Leaf fetch (octree_fsh.c:218-247); call after step() returned kLeaf.
  __device__ __forceinline__ void leaf(const DevScene& sc, int32_t& ms, int32_t& md, float4& col, float4& nrm) {
    ms = load_model(sc.tree[0], ns, level, oob);
    md = DYN ? load_model(sc.tree[1], nd, level, oob) : 0;
    load_attr(sc.model[0], ms, col, nrm, oob);
    if (DYN && md > 0) load_attr(sc.model[1], md, col, nrm, oob);
  }
};

}  // namespace qbc
