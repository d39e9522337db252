// Launchers of the two-level column sweeps (sc_col.cuh), one set per precision
// and size of sc_sweep_sizes.h.
#pragma once
#include "sc_internal.h"
#include "sc_sweep_sizes.h"

namespace sc {

template <typename R, int N> struct ColSweep {
  static void init();  // shared-memory limits, before any launch or capture
  static void launch(bool inv, const ColArgs& a, const void* tw, cudaStream_t st);
};

// false: N has no such sweep (sizes below 32)
template <typename R> bool col_init(int N);
template <typename R> bool col_sweep(int N, bool inv, const ColArgs& a, const void* tw, cudaStream_t st);

}  // namespace sc
