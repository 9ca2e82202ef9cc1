// Lanes without a ray take over part of another lane's walk (rays_kernel).
//
// A few rays end when the longest of them ends: a step is two dependent reads
// and some 300 instructions, a ray up to several hundred steps, and the lanes
// beside it have nothing to do. The entries a walk has listed but not taken
// are independent of what it does before it comes back to them, so a free
// lane can take those of the walk's topmost unfinished level, which the
// shader's order visits last, with a copy of the stack down to that level.
//
// The parts of a ray form a chain in the shader's order: its owner, then the
// lane that took entries from it last, and so on (a lane that takes from
// another is put right behind it). The ray's result is that of the first part
// that ends in a leaf, with every part before it ended without one: a part
// that ends without one is taken out of the chain, one that ends in a leaf
// frees all after it, and an owner that ends without one goes on as its next
// part, whose state it copies. The parts up to that leaf visit exactly the
// nodes that one lane's walk visits, so leaves, entry points and, added up,
// visit counts are the same.
//
// Rays in a 1M-point room, results left on the device, without and with: 1000
// rays 112 -> 48 us a call, 30000 143 -> 81, 1M 0.89 -> 0.75 ms (there only
// the end of the launch shares).
//
// render_kernel does not share: its launches end within a few per cent of
// full use (a 320x240 frame 128.6 -> 125.0 us), and the vote on who waits cost
// a batch of views 0.9 % and two-tree views 2.6 %.
#pragma once

#include "walker_fast.cuh"

namespace qbc {

constexpr int kNoLane = 32;
enum LaneKind : int { kLaneFree, kLaneOwner, kLaneHelper };

// One round, by all lanes of a warp: settles the chains, then free lanes take
// parts of running walks. A free or helping lane's walker and stack column are
// overwritten, an owner's kind is kept. `next` is the lane of the chain's next
// part, `behind` (INSTR) the visits of the parts between the lane's and that
// one, which ended without a leaf (they count unless the lane's ends in one).
// take_ray(src, mine) is called by all lanes: where mine, the lane works on
// src's ray from now on.
template <bool DYN, bool INSTR, class Take>
__device__ __forceinline__ void share_walks(FastWalker<DYN, INSTR>& w, const Stack& st, int maxlevel, int& kind,
                                            bool& running, int& result, int& next, uint2& behind, Take take_ray) {
  constexpr unsigned kAll = 0xFFFFFFFFu;
  constexpr int kWords = FastWalker<DYN, INSTR>::kWords;
  const int lane = threadIdx.x & 31;
  const unsigned bit = 1u << lane;
  auto copy_levels = [&](int src, int levels) {
    const uint32_t* from = st.base + (src - lane);
    for (int k = 0; k < levels * kWords; ++k) st.base[k * st.stride] = from[k * st.stride];
  };
  // the walk's state down to its current cube
  auto copy_path = [&](int src, bool mine) {
    const uint32_t X = __shfl_sync(kAll, w.X, src), Y = __shfl_sync(kAll, w.Y, src), Z = __shfl_sync(kAll, w.Z, src);
    if (mine) {
      w.X = X;
      w.Y = Y;
      w.Z = Z;
    }
  };
  __syncwarp();  // the stacks as the walks left them
  if (__any_sync(kAll, kind == kLaneHelper)) {
    // (a chain has at most 32 parts)
    const unsigned found = __ballot_sync(kAll, kind != kLaneFree && !running && result == kLeaf);
    if (found) {
      unsigned cut = 0u;
      for (int k = 0; k < 32; ++k) {
        const unsigned c =
            __reduce_or_sync(kAll, next != kNoLane && ((found | cut) & bit) ? 1u << (next & 31) : 0u);
        if ((c & ~cut) == 0u) break;
        cut |= c;
      }
      if ((found | cut) & bit) next = kNoLane;
      if (cut & bit) {
        kind = kLaneFree;
        running = false;
      }
    }
    const unsigned missed = __ballot_sync(kAll, kind == kLaneHelper && !running && result != kLeaf);
    if (missed) {
      for (int k = 0; k < 32; ++k) {
        const bool skip = next != kNoLane && ((missed >> (next & 31)) & 1u);
        if (!__any_sync(kAll, skip)) break;
        const int n = __shfl_sync(kAll, next, next & 31);
        if (INSTR) {
          const uint32_t vs = __shfl_sync(kAll, w.vis_s + behind.x, next & 31),
                         vd = __shfl_sync(kAll, w.vis_d + behind.y, next & 31);
          if (skip) behind = make_uint2(behind.x + vs, behind.y + vd);
        }
        if (skip) next = n;
      }
      if (missed & bit) {
        kind = kLaneFree;
        next = kNoLane;
      }
    }
    const bool go_on = kind == kLaneOwner && !running && next != kNoLane;
    const unsigned given = __reduce_or_sync(kAll, go_on ? 1u << (next & 31) : 0u);
    if (given) {
      const int src = go_on ? next & 31 : lane;
      copy_path(src, go_on);
      if (INSTR) {
        const uint32_t vs = __shfl_sync(kAll, w.vis_s, src), vd = __shfl_sync(kAll, w.vis_d, src);
        const uint32_t bs = __shfl_sync(kAll, behind.x, src), bd = __shfl_sync(kAll, behind.y, src);
        if (go_on) {
          w.vis_s += behind.x + vs;
          w.vis_d += behind.y + vd;
          behind = make_uint2(bs, bd);
        }
      }
      const uint32_t more = __shfl_sync(kAll, w.more, src);
      const int level = __shfl_sync(kAll, w.level, src), ns = __shfl_sync(kAll, w.ns, src),
                nd = __shfl_sync(kAll, w.nd, src), r = __shfl_sync(kAll, result, src),
                n = __shfl_sync(kAll, next, src);
      const int flags = __shfl_sync(kAll, (w.slow ? 1 : 0) | (running ? 2 : 0), src);
      if (go_on) {
        copy_levels(src, maxlevel);
        w.more = more;
        w.level = level;
        w.ns = ns;
        w.nd = nd;
        w.slow = flags & 1;
        running = (flags & 2) != 0;
        result = r;
        next = n;
      }
      __syncwarp();
      if (given & bit) {
        kind = kLaneFree;
        running = false;
        next = kNoLane;
      }
    }
  }
  if (INSTR && kind == kLaneOwner && !running) {
    if (result != kLeaf) {
      w.vis_s += behind.x;
      w.vis_d += behind.y;
    }
    behind = make_uint2(0u, 0u);
  }
  // the k-th free lane takes from the k-th walk with entries left
  const unsigned free = __ballot_sync(kAll, kind == kLaneFree), can = __ballot_sync(kAll, running && w.more != 0u);
  const int pairs = min(__popc(free), __popc(can));
  if (pairs == 0) return;
  unsigned lt;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
  const int rf = __popc(free & lt), rc = __popc(can & lt);
  const bool thief = (free & bit) && rf < pairs, victim = (can & bit) && rc < pairs;
  unsigned m = thief ? can : free;
  for (int k = thief ? rf : (victim ? rc : 0); k > 0; --k) m &= m - 1u;
  const int mate = thief || victim ? __ffs((int)m) - 1 : lane;
  copy_path(mate, thief);
  const uint32_t more = __shfl_sync(kAll, w.more, mate);
  const float px = __shfl_sync(kAll, w.p.x, mate), py = __shfl_sync(kAll, w.p.y, mate),
              pz = __shfl_sync(kAll, w.p.z, mate);
  const float ix = __shfl_sync(kAll, w.inv.x, mate), iy = __shfl_sync(kAll, w.inv.y, mate),
              iz = __shfl_sync(kAll, w.inv.z, mate);
  const uint32_t mode = __shfl_sync(kAll, w.mode, mate), sx = __shfl_sync(kAll, w.selx, mate),
                 sy = __shfl_sync(kAll, w.sely, mate), sz = __shfl_sync(kAll, w.selz, mate);
  const float guard = __shfl_sync(kAll, w.guard, mate);
  const int n = __shfl_sync(kAll, next, mate);
  uint2 b = make_uint2(0u, 0u);
  if (INSTR) b = make_uint2(__shfl_sync(kAll, behind.x, mate), __shfl_sync(kAll, behind.y, mate));
  take_ray(mate, thief);
  if (thief) {
    // A walk at maxlevel lists nothing and takes the next entry that is left:
    // one of the level taken over.
    const int l = __ffs((int)more) - 1;
    copy_levels(mate, l + 1);
    w.more = 1u << l;
    w.p = make_float3(px, py, pz);
    w.inv = make_float3(ix, iy, iz);
    w.mode = mode;
    w.selx = sx;
    w.sely = sy;
    w.selz = sz;
    w.guard = guard;
    w.level = maxlevel;
    w.ns = 0;
    w.nd = 0;
    w.slow = false;
    w.oob = false;
    w.vis_s = 0;
    w.vis_d = 0;
    w.target = 0u;
    w.tdepth = 0;
    kind = kLaneHelper;
    running = true;
    result = kRunning;
    next = n;
    behind = b;
  }
  __syncwarp();
  if (victim) {
    behind = make_uint2(0u, 0u);
    w.more &= w.more - 1u;
    next = mate;
  }
}

}  // namespace qbc
