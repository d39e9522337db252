// Dispatch of the column sweeps over precision and size (sc_col.h).
#include "sc_col.h"

namespace sc {

template <typename R> bool col_init(int N) {
  switch (N) {
#define SC_CASE(NN, ...) case NN: ColSweep<R, NN>::init(); break;
    SC_SWEEP_SIZES(SC_CASE)
#undef SC_CASE
    default: return true;
  }
  return cudaGetLastError() == cudaSuccess;
}

template <typename R> bool col_sweep(int N, bool inv, const ColArgs& a, const void* tw, cudaStream_t st) {
  switch (N) {
#define SC_CASE(NN, ...) case NN: ColSweep<R, NN>::launch(inv, a, tw, st); return true;
    SC_SWEEP_SIZES(SC_CASE)
#undef SC_CASE
    default: return false;
  }
}

template bool col_init<float>(int);
template bool col_init<double>(int);
template bool col_sweep<float>(int, bool, const ColArgs&, const void*, cudaStream_t);
template bool col_sweep<double>(int, bool, const ColArgs&, const void*, cudaStream_t);

}  // namespace sc
