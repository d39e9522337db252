// Launchers of the warp-per-row-pair x sweeps (sc_xrow.cuh), one set per
// precision and size of sc_sweep_sizes.h.
#pragma once
#include "sc_internal.h"
#include "sc_sweep_sizes.h"

namespace sc {

template <typename R, int N> struct XRow {
  static void init();  // shared-memory limits, before any launch or capture
  static void ns(const XArgs& a, const void* tx, cudaStream_t st);
  static void c2r(const XPlainArgs& a, const void* tx, cudaStream_t st);
  static void r2c(const XPlainArgs& a, const void* tx, cudaStream_t st);
  static void point(const XPointArgs& a, const void* tx, cudaStream_t st);
  static void vmax(const XPlainArgs& a, const void* tx, unsigned long long* out, cudaStream_t st);
};

// false: N has no such sweep (sizes below 32), or the call is not one it takes
template <typename R> bool xrow_init(int N);
template <typename R> bool xrow_ns(int N, const XArgs& a, const void* tw, cudaStream_t st);
template <typename R> bool xrow_c2r(int N, const XPlainArgs& a, const void* tw, cudaStream_t st);
template <typename R> bool xrow_r2c(int N, const XPlainArgs& a, const void* tw, cudaStream_t st);
template <typename R> bool xrow_point(int N, const XPointArgs& a, const void* tw, cudaStream_t st);
template <typename R>
bool xrow_vmax(int N, const XPlainArgs& a, const void* tw, unsigned long long* out, cudaStream_t st);

}  // namespace sc
