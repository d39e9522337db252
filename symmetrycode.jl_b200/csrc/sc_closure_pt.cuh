// Point functions of the classical closures, shared by the pointwise kernels
// (sc_les.cu) and the fused x sweeps (sc_xrow.cuh).
#pragma once
#include <math.h>

#include "sc_les.h"

namespace sc {

// clark_kernel! / smagorinsky_kernel! / verstappen_kernel! (src/closures.jl:37-62):
// velocity gradient G -> stress t; d2 = Delta^2, p0 = C_s or C
template <typename R, int D>
__device__ __forceinline__ void closure_point(int kind, R d2, R p0, const R G[3][3], R t[3][3]) {
  if (kind == kClark) {
    for (int p = 0; p < D; ++p)
      for (int q = 0; q < D; ++q) {
        R s = 0;
        for (int k = 0; k < D; ++k) s += G[p][k] * G[q][k];
        t[p][q] = d2 / R(12) * s;
      }
  } else {
    R S[3][3];
    R ss = 0;
    for (int p = 0; p < D; ++p)
      for (int q = 0; q < D; ++q) {
        S[p][q] = (G[p][q] + G[q][p]) / R(2);
        ss += S[p][q] * S[p][q];
      }
    R nu;
    if (kind == kSmagorinsky) {
      const R cs = p0;
      nu = cs * cs * d2 * sqrt(R(2) * ss);
    } else {  // Verstappen: q = tr(S S)/2, r = tr(S S S)/3, nu = C^2 Delta^2 |r| / q
      R SS[3][3];
      for (int p = 0; p < 3; ++p)
        for (int q = 0; q < 3; ++q) {
          R s = 0;
          for (int k = 0; k < 3; ++k) s += S[p][k] * S[k][q];
          SS[p][q] = s;
        }
      R trss = 0, trsss = 0;
      for (int p = 0; p < 3; ++p) {
        trss += SS[p][p];
        for (int k = 0; k < 3; ++k) trsss += SS[p][k] * S[k][p];
      }
      const R qq = trss / R(2), rr = trsss / R(3);
      const R c = p0;
      nu = c * c * d2 * fabs(rr) / qq;
    }
    for (int p = 0; p < D; ++p)
      for (int q = 0; q < D; ++q) t[p][q] = -R(2) * nu * S[p][q];
  }
}

// eddy viscosity of smagorinsky_tensor! (src/closures.jl:117-150) with C_s = 1; s: packed strain rate
template <typename R, int D> __device__ __forceinline__ R smag_viscosity(R d2, const R s[6]) {
  constexpr int NP = D == 3 ? 6 : 3;
  R s2 = 0;
  for (int q = 0; q < D; ++q) s2 += s[q] * s[q];
  for (int q = D; q < NP; ++q) s2 += R(2) * s[q] * s[q];
  return d2 * sqrt(R(2) * s2);
}

}  // namespace sc
