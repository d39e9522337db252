// Sizes of the two-level register sweeps and how each length is split.
//
// X(N, xf1, xf2, xd1, xd2, cf1, cf2, cd1, cd2): N = xf1 * xf2 splits the x rows
// in FP32 (xf1 lanes of a warp hold xf2 points each between the inverse and the
// forward transform), N = xd1 * xd2 in FP64, N = cf1 * cf2 the column sweeps in
// FP32 (radix cf1 first), N = cd1 * cd2 in FP64.
// x rows: few points a lane keep the slots small (32 / xf1 row pairs
// a warp, 4 to 9 slots each) and more warps resident, which is worth more than
// full rounds of work items: 128 FP32, product sweep of 2 GB 743 us as 8 x 16 and
// 578 as 16 x 8, Clark's closure sweep 54 and 38 us; 256 FP64 625 us as 16 x 16
// and 570 as 32 x 8; 120 FP32 801 us as 8 x 15 and 632 as 15 x 8.  Below that the
// sweeps of a grid are short and the wider split starts faster (64 FP32, 64^3:
// 5.8 us as 8 x 8, 5.1 as 16 x 4).
// Columns: the narrow radix first.  It gathers from global memory, so more threads
// each keep fewer addresses and loads, and the wide one reads shared memory only;
// pruned outputs are left out in finer steps.  y forward / z forward sweep, FP64:
// 512 415 / 235 us as 32 x 16 and 259 / 149 as 16 x 32, 540 382 / 262 as 27 x 20 and
// 292 / 191 as 20 x 27, 320 329 / 45 and 282 / 38; FP32: 384 389 / 47 as 24 x 16 and
// 323 / 39 as 16 x 24; small sizes gain 0 to 15 %.  The exceptions: 540 FP32 (166 /
// 109 us as 27 x 20, 170 / 113 as 20 x 27) and 128, where in FP32 sc_fast.cu has both
// as variants and the right-hand side of the network keeps the rounding of this one.
// Sizes below 32 keep the shared-memory engine of sc_kernels.cu.
#pragma once

#define SC_SWEEP_SIZES_A(X) \
  X(32, 16, 2, 16, 2, 4, 8, 4, 8) X(36, 12, 3, 12, 3, 6, 6, 6, 6) X(40, 20, 2, 20, 2, 5, 8, 5, 8) \
  X(48, 12, 4, 12, 4, 6, 8, 6, 8) X(60, 15, 4, 15, 4, 6, 10, 6, 10) X(64, 16, 4, 16, 4, 8, 8, 8, 8) \
  X(72, 18, 4, 18, 4, 8, 9, 8, 9) X(80, 16, 5, 16, 5, 8, 10, 8, 10) X(90, 15, 6, 15, 6, 9, 10, 9, 10) \
  X(96, 16, 6, 16, 6, 8, 12, 8, 12)
#define SC_SWEEP_SIZES_B(X) \
  X(120, 15, 8, 15, 8, 10, 12, 10, 12) X(128, 16, 8, 16, 8, 16, 8, 16, 8) X(160, 20, 8, 20, 8, 10, 16, 10, 16) \
  X(180, 20, 9, 20, 9, 12, 15, 12, 15) X(192, 24, 8, 24, 8, 12, 16, 12, 16) X(240, 30, 8, 30, 8, 15, 16, 15, 16) \
  X(256, 32, 8, 32, 8, 16, 16, 16, 16)
#define SC_SWEEP_SIZES_C(X) \
  X(270, 30, 9, 27, 10, 15, 18, 15, 18) X(320, 32, 10, 32, 10, 16, 20, 16, 20) X(360, 24, 15, 24, 15, 18, 20, 18, 20) \
  X(384, 24, 16, 24, 16, 16, 24, 16, 24) X(512, 32, 16, 32, 16, 16, 32, 16, 32)
#define SC_SWEEP_SIZES_D(X) \
  X(540, 30, 18, 30, 18, 27, 20, 20, 27) X(640, 32, 20, 32, 20, 20, 32, 20, 32) X(720, 30, 24, 30, 24, 24, 30, 24, 30) \
  X(768, 32, 24, 32, 24, 24, 32, 24, 32) X(810, 30, 27, 30, 27, 27, 30, 27, 30) X(1024, 32, 32, 32, 32, 32, 32, 32, 32)
#define SC_SWEEP_SIZES(X) SC_SWEEP_SIZES_A(X) SC_SWEEP_SIZES_B(X) SC_SWEEP_SIZES_C(X) SC_SWEEP_SIZES_D(X)

namespace sc {

template <typename R, int N> struct XSplit;  // lanes N1, points per lane N2
template <typename R, int N> struct CSplit;  // first radix N1, second radix N2
#define SC_SPLIT(N, A1, A2, B1, B2, C1, C2, D1, D2) \
  template <> struct XSplit<float, N> { static constexpr int N1 = A1, N2 = A2; }; \
  template <> struct XSplit<double, N> { static constexpr int N1 = B1, N2 = B2; }; \
  template <> struct CSplit<float, N> { static constexpr int N1 = C1, N2 = C2; }; \
  template <> struct CSplit<double, N> { static constexpr int N1 = D1, N2 = D2; }; \
  static_assert(A1 * A2 == N && B1 * B2 == N && C1 * C2 == N && D1 * D2 == N && A1 <= 32 && B1 <= 32, "split of N");
SC_SWEEP_SIZES(SC_SPLIT)
#undef SC_SPLIT

// sizes with two-level sweeps; xn1 / xn2: the x split (for the host's twiddle tables)
inline bool sweep_size(int n, bool f32, int* xn1 = nullptr, int* xn2 = nullptr) {
  switch (n) {
#define SC_CASE(N, A1, A2, B1, B2, C1, C2, D1, D2) \
  case N: if (xn1) { *xn1 = f32 ? A1 : B1; *xn2 = f32 ? A2 : B2; } return true;
    SC_SWEEP_SIZES(SC_CASE)
#undef SC_CASE
    default: return false;
  }
}

// Rows of one launch of a product sweep whose rows are `len` elements long: whole
// row pairs, and few enough that the kernels' 32-bit element indexes (those of a last
// warp that is partly empty included) stay below 2^31.  A plan's n^2 rows always are
// (n <= 1024); the microbenchmark takes any number.
inline long long sweep_rows(long long len) { return (2147483647LL / len - 64) & ~1LL; }

// the smallest of these sizes that is at least m (0: none)
inline int sweep_size_from(int m) {
#define SC_CASE(N, ...) if (N >= m) return N;
  SC_SWEEP_SIZES(SC_CASE)
#undef SC_CASE
  return 0;
}

}  // namespace sc
