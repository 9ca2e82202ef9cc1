// Whether the creator tables of the dynamic tree's builds (build.cu) are empty
// on the device, as a build leaves them and the next one expects them.
#pragma once

namespace qbc {

struct TableState {
  bool empty = false;

  // The arrays are new, their contents unknown.
  void replaced() { empty = false; }

  // A build's launches begin (`uses`: it is one with creator tables). True
  // where they must empty the tables first. Until end() the tables count as
  // not empty: a build may stop midway.
  bool begin(bool uses) {
    const bool reset = uses && !empty;
    if (uses) empty = false;
    return reset;
  }

  // All is queued, in a build that began with `reset`. Only a build with
  // tables leaves them empty, and not where its emptying was recorded for a
  // graph instead of run.
  void end(bool uses, bool reset, bool captured) {
    if (uses && !(reset && captured)) empty = true;
  }
};

}  // namespace qbc
