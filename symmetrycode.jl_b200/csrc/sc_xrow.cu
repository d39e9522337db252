// Dispatch of the x sweeps over precision and size (sc_xrow.h).
#include "sc_fft.cuh"
#include "sc_xrow.h"

namespace sc {

// the x tables of a plan's twiddle buffer (t1, then t2)
template <typename R> static const void* xtab(int N, const void* tw) {
  return static_cast<const char*>(tw) + twiddle_x_offset(N, sizeof(typename V2<R>::T));
}

template <typename R> bool xrow_init(int N) {
  switch (N) {
#define SC_CASE(NN, ...) case NN: XRow<R, NN>::init(); break;
    SC_SWEEP_SIZES(SC_CASE)
#undef SC_CASE
    default: return true;
  }
  return cudaGetLastError() == cudaSuccess;
}

// every caller's rows come in pairs (N is even) and indexes fit 32 bits (N <= 1024);
// inputs of the product sweep and of vmax are compact rows of N / 3 + 1 modes,
// or, in 3D with at most N / 5 + 1 modes kept, longer rows of fewer than N / 2 + 1
template <typename R> bool xrow_ns(int N, const XArgs& a, const void* tw, cudaStream_t st) {
  const bool wide = a.D == 3 && a.K1in > N / 3 + 1 && 2 * (a.K1in - 1) < N && a.K1out <= N / 5 + 1;
  if ((a.K1in != N / 3 + 1 && !wide) || a.K1out > a.K1in || (a.nrows & 1)) return false;
  switch (N) {
#define SC_CASE(NN, ...) case NN: XRow<R, NN>::ns(a, xtab<R>(N, tw), st); return true;
    SC_SWEEP_SIZES(SC_CASE)
#undef SC_CASE
    default: return false;
  }
}
template <typename R> bool xrow_c2r(int N, const XPlainArgs& a, const void* tw, cudaStream_t st) {
  if ((a.K1 != N / 3 + 1 && a.K1 != N / 2 + 1) || (a.nrows & 1)) return false;
  switch (N) {
#define SC_CASE(NN, ...) case NN: XRow<R, NN>::c2r(a, xtab<R>(N, tw), st); return true;
    SC_SWEEP_SIZES(SC_CASE)
#undef SC_CASE
    default: return false;
  }
}
template <typename R> bool xrow_r2c(int N, const XPlainArgs& a, const void* tw, cudaStream_t st) {
  if ((a.K1 != N / 3 + 1 && a.K1 != N / 2 + 1) || (a.nrows & 1)) return false;
  switch (N) {
#define SC_CASE(NN, ...) case NN: XRow<R, NN>::r2c(a, xtab<R>(N, tw), st); return true;
    SC_SWEEP_SIZES(SC_CASE)
#undef SC_CASE
    default: return false;
  }
}
template <typename R> bool xrow_point(int N, const XPointArgs& a, const void* tw, cudaStream_t st) {
  if ((a.nin != 6 && a.nin != 9) || (a.nrows & 1)) return false;
  switch (N) {
#define SC_CASE(NN, ...) case NN: XRow<R, NN>::point(a, xtab<R>(N, tw), st); return true;
    SC_SWEEP_SIZES(SC_CASE)
#undef SC_CASE
    default: return false;
  }
}
template <typename R>
bool xrow_vmax(int N, const XPlainArgs& a, const void* tw, unsigned long long* out, cudaStream_t st) {
  if (a.K1 != N / 3 + 1 || (a.nrows & 1)) return false;
  switch (N) {
#define SC_CASE(NN, ...) case NN: XRow<R, NN>::vmax(a, xtab<R>(N, tw), out, st); return true;
    SC_SWEEP_SIZES(SC_CASE)
#undef SC_CASE
    default: return false;
  }
}

#define SC_INST(R)                                                                                      \
  template bool xrow_init<R>(int);                                                                      \
  template bool xrow_ns<R>(int, const XArgs&, const void*, cudaStream_t);                               \
  template bool xrow_c2r<R>(int, const XPlainArgs&, const void*, cudaStream_t);                         \
  template bool xrow_r2c<R>(int, const XPlainArgs&, const void*, cudaStream_t);                         \
  template bool xrow_point<R>(int, const XPointArgs&, const void*, cudaStream_t);                       \
  template bool xrow_vmax<R>(int, const XPlainArgs&, const void*, unsigned long long*, cudaStream_t);
SC_INST(float)
SC_INST(double)
#undef SC_INST

}  // namespace sc
