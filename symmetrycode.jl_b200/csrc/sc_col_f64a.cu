// Column sweeps of one precision and group of sizes (one object each, so that they compile in parallel).
#include "sc_col.cuh"

namespace sc {
#define SC_CASE(N, ...) template struct ColSweep<double, N>;
SC_SWEEP_SIZES_A(SC_CASE)
#undef SC_CASE
}  // namespace sc
