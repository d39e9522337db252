// Column sweeps of one precision and group of sizes (one object each, so that they compile in parallel).
#include "sc_col.cuh"

namespace sc {
#define SC_CASE(N, ...) template struct ColSweep<float, N>;
SC_SWEEP_SIZES_B(SC_CASE)
#undef SC_CASE
}  // namespace sc
