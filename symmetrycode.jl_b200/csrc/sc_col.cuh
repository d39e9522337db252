// Two-level register FFT column sweeps (sm_100a), FP32 and FP64, every size of
// sc_sweep_sizes.h.
//
// A length-N transform along a strided axis is split N = N1 N2:
//   step 1  thread (kx of the tile, j < N2) gathers x[N2 n1 + j], n1 < N1,
//           straight from global memory into registers, runs a radix-N1 DFT,
//           multiplies by exp(-+2 pi i j k1 / N) and writes one row of the
//           shared exchange buffer;
//   step 2  thread (kx, k1) reads the N2 values of its column, runs a radix-N2
//           DFT and stores X[k1 + N1 k2] straight to global memory (pruned to
//           the retained modes on the forward side).
// Each element crosses shared memory once, and every thread keeps N1
// independent global loads in flight.
#pragma once
#include "sc_fft.cuh"
#include "sc_col.h"

namespace sc {

// T consecutive kx per tile; S = 1 transposes the split (N2 first)
template <typename R, int N, int T, int S = 0> struct Col2Cfg {
  using C = typename V2<R>::T;
  static constexpr int N1 = S ? CSplit<R, N>::N2 : CSplit<R, N>::N1, N2 = S ? CSplit<R, N>::N1 : CSplit<R, N>::N2;
  static constexpr int NJ = N1 > N2 ? N1 : N2;
  static constexpr int NT = T * NJ;
  static constexpr int SR = N2 * T + 8;  // exchange row stride (+8: half-bank shift between rows)
  static constexpr size_t SMEM = size_t(N1) * SR * sizeof(C);
  // resident CTAs: what shared memory and the registers of the wider radix in
  // flight allow, plus 40 (FP32) or 56 (FP64) for addresses and temporaries (56
  // in FP32: 540 y inverse 105 us instead of 88; 40 in FP64: spills, 640 y
  // inverse 232 us instead of 192); 810 FP32: 80 registers, three CTAs at T = 8
  static constexpr int RG = 2 * NJ * int(sizeof(R) / 4) + (sizeof(R) == 4 ? 40 : 56), REGS = RG > 255 ? 255 : (RG + 7) / 8 * 8;
  static constexpr int BR = 65536 / ((NT + 31) / 32 * 32 * REGS), BS = int((227 * 1024) / (SMEM + 1024));
  static constexpr int BB = BR < BS ? BR : BS;
  static constexpr bool F810 = N == 810 && sizeof(R) == 4, F2N = sizeof(R) == 4 && (N == 64 || N == 128 || N == 256);
  static constexpr int MINB = F810 ? (T == 4 ? 6 : (T == 8 ? 3 : 1)) : F2N || BB < 1 ? 1 : (BB > 16 ? 16 : BB);
};

// FULL: the transform axis has the 2/3-rule compact layout of the solver
// (kpos = N/3 + 1, kneg = N/3), so which of each thread's N1 gathers (inverse)
// or N2 stores (forward) touch a retained mode is known at compile time except
// in the one block that straddles a boundary; the unused forward outputs are
// then never formed.
// FILT: the gather multiplies by ColArgs::wtab (a closure's test filter).
template <typename R, int N, int T, bool INV, bool FULL, int S = 0, bool FILT = false>
__global__ void __launch_bounds__(Col2Cfg<R, N, T, S>::NT, Col2Cfg<R, N, T, S>::MINB)
k_col2(const __grid_constant__ ColArgs a, const typename V2<R>::T* __restrict__ tw) {
  using C = typename V2<R>::T;
  using Cfg = Col2Cfg<R, N, T, S>;
  constexpr int N1 = Cfg::N1, N2 = Cfg::N2, SR = Cfg::SR;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C* ys = reinterpret_cast<C*>(smem_raw);
  const int t = threadIdx.x % T, j = threadIdx.x / T;
  const int kx = blockIdx.x * T + t;
  const int c = blockIdx.y;
  const C* __restrict__ in = static_cast<const C*>(a.in[blockIdx.z]);
  C* __restrict__ out = static_cast<C*>(a.out[blockIdx.z]);
  const bool live = kx < a.K1;
  constexpr int KP = N / 3 + 1, KN = N / 3;
  const int kpos = FULL ? KP : a.kpos, kneg = FULL ? KN : a.kneg;
  const int Kc = kpos + kneg;
  // element offsets fit in 32 bits for every sweep (at most ~5.4e8 elements
  // per component), so the per-element address arithmetic stays 32-bit
  const int ies = int(a.in_es), oes = int(a.out_es);
  if (j < N2) {
    C v[N1];
    const C* base = in + kx + (long long)c * a.in_cs;
    if (INV) {
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1) {
        const int e = N2 * n1 + j;
        v[n1] = mk<C>(R(0), R(0));
        const int rg = FULL ? crange(N2 * n1, N2, N, KP, KN) : 3;
        if (rg == 2) continue;
        const int p = rg == 0 ? e : (rg == 1 ? e - N + Kc : cpos(e, N, kpos, kneg));
        if (live && p >= 0 && !(a.zero_origin && kx == 0 && c == 0 && p == 0)) {
          v[n1] = __ldg(base + p * ies);
          if constexpr (FILT) {
            const int ke = p < kpos ? p : p - Kc, kc = c < kpos ? c : c - Kc;
            const R w = __ldg(static_cast<const R*>(a.wtab) + kx * kx + kc * kc + ke * ke);
            v[n1] = mk<C>(w * v[n1].x, w * v[n1].y);
          }
        }
      }
    } else {
      const C* bj = base + j * ies;
      const int st = N2 * ies;
#pragma unroll
      for (int n1 = 0; n1 < N1; ++n1) v[n1] = live ? __ldg(bj + n1 * st) : mk<C>(R(0), R(0));
    }
    DFT<N1, INV, C>::run(v);
#pragma unroll
    for (int k1 = 1; k1 < N1; ++k1) {
      C w = __ldg(&tw[j * k1]);
      if (INV) w.y = -w.y;
      v[k1] = cmul(v[k1], w);
    }
#pragma unroll
    for (int k1 = 0; k1 < N1; ++k1) ys[k1 * SR + j * T + t] = v[k1];
  }
  __syncthreads();
  if (j < N1 && live) {
    C w[N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) w[n2] = ys[j * SR + n2 * T + t];
    DFT<N2, INV, C>::run(w);
    C* obase = out + kx + (long long)c * a.out_cs;
    if (INV) {
      C* oj = obase + j * oes;
      const int st = N1 * oes;
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) oj[k2 * st] = w[k2];
    } else {
      // retained e = j + N1 k2: e < kpos keeps its index, e >= N - kneg moves down by N - Kc
      const int shift = N - Kc;
#pragma unroll
      for (int k2 = 0; k2 < N2; ++k2) {
        const int e = j + N1 * k2;
        const int rg = FULL ? crange(N1 * k2, N1, N, KP, KN) : 3;
        if (rg == 0) obase[e * oes] = w[k2];
        else if (rg == 1) obase[(e - shift) * oes] = w[k2];
        else if (rg == 3) {
          if (e < kpos) obase[e * oes] = w[k2];
          else if (e >= N - kneg) obase[(e - shift) * oes] = w[k2];
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// launcher of one precision and size
// ---------------------------------------------------------------------------
// Tile width: FP32 16 kx (128-byte rows) up to 128, 8 from 160 on, where the
// smaller tile's extra CTAs per SM gain more than the wider rows (384, y
// inverse: 242 us at 16, 182 at 8; 120, y forward: 10 and 12); FP64 8 kx
// (128-byte rows) up to 384, 4 beyond (384, y inverse: 300 us at 8, 322 at 4;
// 540: 231 and 193)
template <typename R, int N> struct ColTile {
  static constexpr int T = sizeof(R) == 4 ? (N <= 128 ? 16 : 8) : (N <= 384 ? 8 : 4);
};

template <typename R, int N> void ColSweep<R, N>::init() {
  constexpr int T = ColTile<R, N>::T;
  constexpr size_t b = Col2Cfg<R, N, T>::SMEM;
  if (b > 48 * 1024) {
    cudaFuncSetAttribute(k_col2<R, N, T, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(b));
    cudaFuncSetAttribute(k_col2<R, N, T, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(b));
    cudaFuncSetAttribute(k_col2<R, N, T, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(b));
    cudaFuncSetAttribute(k_col2<R, N, T, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(b));
    cudaFuncSetAttribute(k_col2<R, N, T, true, true, 0, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(b));
  }
}

template <typename R, int N> void ColSweep<R, N>::launch(bool inv, const ColArgs& a, const void* tw, cudaStream_t st) {
  constexpr int T = ColTile<R, N>::T;
  using C = typename V2<R>::T;
  using Cfg = Col2Cfg<R, N, T>;
  const dim3 grid((a.K1 + T - 1) / T, a.ncols, a.ncomp);
  const C* t2 = static_cast<const C*>(tw);
  const bool full = a.kpos == N / 3 + 1 && a.kneg == N / 3;
  if (inv && full && a.wtab) k_col2<R, N, T, true, true, 0, true><<<grid, Cfg::NT, Cfg::SMEM, st>>>(a, t2);
  else if (inv && full) k_col2<R, N, T, true, true><<<grid, Cfg::NT, Cfg::SMEM, st>>>(a, t2);
  else if (inv) k_col2<R, N, T, true, false><<<grid, Cfg::NT, Cfg::SMEM, st>>>(a, t2);
  else if (full) k_col2<R, N, T, false, true><<<grid, Cfg::NT, Cfg::SMEM, st>>>(a, t2);
  else k_col2<R, N, T, false, false><<<grid, Cfg::NT, Cfg::SMEM, st>>>(a, t2);
}

}  // namespace sc
