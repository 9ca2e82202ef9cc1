// Numbers of the render kernels' template instances, one each: a context
// remembers by them which instances' attributes it has set.
#pragma once

namespace qbc {

constexpr int kWalkKinds = 3;                      // render.cuh: Walk
constexpr int kModeKinds = 5;                      // render.cuh: Mode
constexpr int kPerWalk = 4 * (kModeKinds + 1);     // ... and the shade pass with proposals
constexpr int kRenderKernels = kPerWalk * kWalkKinds;
constexpr int kKernels = kRenderKernels + 4;       // with simple_kernel's

// render_kernel<exact, dyn, mode, prop, walk>; only a shade pass has prop.
constexpr int render_kernel_index(bool exact, bool dyn, int mode, bool prop, int walk) {
  return (exact ? 1 : 0) + (dyn ? 2 : 0) + 4 * (prop ? kModeKinds : mode) + kPerWalk * walk;
}

// simple_kernel<exact, dyn>
constexpr int simple_kernel_index(bool exact, bool dyn) {
  return kRenderKernels + (exact ? 1 : 0) + (dyn ? 2 : 0);
}

}  // namespace qbc
