// x sweeps, one warp per group of row pairs (sm_100a): the product sweep of the
// right-hand side, the plain c2r and r2c of batches of fields, and the CFL
// maximum.  FP32 and FP64, every size of sc_sweep_sizes.h.
//
// A real transform of length N = N1 N2 runs on two real rows packed as a + i b
// ("pencil").  The inverse (c2r) takes f = N2 n1 + j:
//   I1  item (pencil, j < N2): gather the N1 Hermitian-extended values from
//       global memory, radix-N1, twiddle exp(+2 pi i j k1 / N)   -> slot [k1][j]
//   I2  lane i < N1: radix-N2 over j: physical x = i + N1 k2, in registers
// and the forward (r2c) is its mirror image, x = i + N1 n, k = k' + N2 m:
//   F1  lane i: radix-N2 over n, twiddle exp(-2 pi i i k' / N)   -> slot [k'][i]
//   F2  item (pencil, k' < N2): radix-N1 over i, retained k only, written back
//       to the N1 slot places the item itself read
//   S   split the packed spectra and store rows.
// I2 leaves every lane with exactly the points its F1 needs, so the products
// are formed in registers.  A warp holds W = 32 / N1 row pairs, so every
// exchange is inside one warp: __syncwarp only, no CTA barrier, and the CTAs
// are just bundles of independent warps.  The slots' row strides (SP, SQ) make
// both sides of every exchange, and the gather of S, nearly free of bank conflicts;
// the twiddles come from tables in the order the lanes read them.
//
// What bounds it: FP32 issue (FP64: the FP64 pipe) at large N with the rows
// streaming from HBM.  Against the CTA-wide kernels it replaces it moves about
// half the shared-memory bytes (47 -> 26 KB a row at N = 256, FP32): 2 GB of rows at
// N = 256 1069 -> 603 us in FP32 and 2687 -> 570 in FP64, at 540 in FP64 1867 -> 905.
#pragma once
#include "sc_fft.cuh"
#include "sc_internal.h"
#include "sc_closure_pt.cuh"
#include "sc_xrow.h"

namespace sc {

template <typename R, int N> struct XRowCfg {
  using C = typename V2<R>::T;
  static constexpr int N1 = XSplit<R, N>::N1, N2 = XSplit<R, N>::N2;
  static constexpr int W = 32 / N1;               // row pairs per warp
  // Slot row strides of the inverse / forward exchange.  Odd ones keep both sides
  // of an exchange free of bank conflicts; S reads 16 / N2 neighbouring values of
  // m for each k' at once, so in FP32 (16 lanes a phase) with N2 = 8 or 4 the
  // forward stride is 2 or 4 times an odd number, and the slot stride odd: k' SQ + m
  // and, over neighbouring pencils, k' SQ + q PS are then distinct modulo 16.
  // Against odd strides everywhere, product sweep of 2 GB of rows, FP32: N = 64 590
  // -> 492 us, 60 564 -> 503, 128 577 -> 564, 256 616 -> 603; 160 to 240 equal.
  static constexpr bool P8 = sizeof(R) == 4 && N2 == 8, P4 = sizeof(R) == 4 && N2 == 4;
  static constexpr int SP = N2 | 1;
  static constexpr int SQ = P8 ? (N1 + 1) / 4 * 4 + 2 : P4 ? (N1 + 3) / 8 * 8 + 4 : N1 | 1;
  static constexpr int PSM = N1 * SP > N2 * SQ ? N1 * SP : N2 * SQ;
  static constexpr int PO = P8 ? 9 : P4 ? 5 : 8;  // = 8 (mod 16) else: two groups of 8 lanes meet no bank twice
  static constexpr int PS = (PSM + 15 - PO) / 16 * 16 + PO;
  static_assert(SQ >= N1 && PS >= PSM, "slot strides");
  static constexpr int KC = N / 3;
  static constexpr size_t slots(int n) { return size_t(n) * W * PS * sizeof(C); }
  // warps per CTA and CTAs per SM for n slots a warp: as many warps as shared
  // memory and `regs` registers a thread allow
  static constexpr int wpc(int n) { return 4 * slots(n) <= 57 * 1024 ? 4 : (2 * slots(n) <= 75 * 1024 ? 2 : 1); }
  static constexpr int minb(int n, int regs) {
    const int a = int((227 * 1024) / (wpc(n) * slots(n) + 1024)), b = 65536 / (regs * 32 * wpc(n));
    const int m = a < b ? a : b;
    return m < 1 ? 1 : (m > 32 / wpc(n) ? 32 / wpc(n) : m);
  }
  static constexpr int rsz = sizeof(R) / 4;
  // the velocities of a row pair stay in the slots instead of registers (3D
  // product sweep): FP64 from 20 points a lane on, where they spilled (810 FP64,
  // 2.0 GB of rows: 1925 us with the spills).  The 2D sweep has registers only and
  // spills 0.2 to 2 KB a thread there; against the shared-memory engine a right-hand
  // side in FP64 takes 26.6 us instead of 42.8 at 640^2, 45.1 instead of 55.9 at 810^2
  // and 51.3 instead of 82.3 at 1024^2
  static constexpr bool IN_SLOTS = rsz * N2 >= 40;
  static constexpr int cap(int r) { return r > 255 ? 255 : (r + 7) / 8 * 8; }
  // registers: a radix in flight (2 per point) or the velocities of a row pair
  // (4 per point) and a pencil
  static constexpr int regs_ns =
      cap(IN_SLOTS || N1 > 3 * N2 ? 2 * (N1 > N2 ? N1 : N2) * rsz + 64 : 6 * N2 * rsz + 48);
  static constexpr int regs_plain = cap(2 * (N1 > N2 ? N1 : N2) * rsz + 64);
};

// Z[f] = A[f] + i B[f] of the half spectra ra, rb (Hermitian extension): mode k
// itself, and mode N - k from its mirror image.  `real`: the mean or the Nyquist
// mode of a real row, whose imaginary part drops out.
template <typename C>
__device__ __forceinline__ C xr_direct(const C* ra, const C* rb, int k, bool real) {
  C x = __ldg(ra + k), y = __ldg(rb + k);
  if (real) { x.y = 0; y.y = 0; }
  return mk<C>(x.x - y.y, x.y + y.x);
}
template <typename C>
__device__ __forceinline__ C xr_mirror(const C* ra, const C* rb, int k) {
  const C x = __ldg(ra + k), y = __ldg(rb + k);
  return mk<C>(x.x + y.y, y.x - x.y);
}

// I1 of one item.  KMAX: highest stored mode (N / 3, or N / 2 for the full RFFT
// layout), so the stored range of each block of N2 indices is known at compile
// time except where it straddles an end.  `live`: the rows exist.
template <typename R, int N, int KMAX>
__device__ __forceinline__ void xr_i1(const typename V2<R>::T* ra, const typename V2<R>::T* rb, bool live, int j,
                                      const typename V2<R>::T* __restrict__ t1, typename V2<R>::T* slot) {
  using C = typename V2<R>::T;
  using Cfg = XRowCfg<R, N>;
  constexpr int N1 = Cfg::N1, N2 = Cfg::N2;
  // modes f <= KMAX are stored, f >= N - KNEG come from the mirror image
  constexpr int KNEG = 2 * KMAX == N ? KMAX - 1 : KMAX;
  C v[N1];
#pragma unroll
  for (int n1 = 0; n1 < N1; ++n1) {
    const int f = N2 * n1 + j;
    const int cls = crange(N2 * n1, N2, N, KMAX + 1, KNEG);
    const bool real = (n1 == 0 && j == 0) ||
                      (2 * KMAX == N && N2 * n1 <= KMAX && KMAX < N2 * n1 + N2 && f == KMAX);
    v[n1] = mk<C>(R(0), R(0));
    if (!live || cls == 2) continue;
    if (cls == 0) v[n1] = xr_direct(ra, rb, f, real);
    else if (cls == 1) v[n1] = xr_mirror(ra, rb, N - f);
    else if (f <= KMAX) v[n1] = xr_direct(ra, rb, f, real);
    else if (f >= N - KNEG) v[n1] = xr_mirror(ra, rb, N - f);
  }
  DFT<N1, true, C>::run(v);
#pragma unroll
  for (int k1 = 1; k1 < N1; ++k1) {
    const C w = __ldg(t1 + k1 * N2 + j);
    v[k1] = cmul(v[k1], mk<C>(w.x, -w.y));
  }
#pragma unroll
  for (int k1 = 0; k1 < N1; ++k1) slot[k1 * Cfg::SP + j] = v[k1];
}

// I2 of lane i: v[k2] = physical values at x = i + N1 k2
template <typename R, int N>
__device__ __forceinline__ void xr_i2(const typename V2<R>::T* slot, int i, typename V2<R>::T* v) {
  using Cfg = XRowCfg<R, N>;
#pragma unroll
  for (int n2 = 0; n2 < Cfg::N2; ++n2) v[n2] = slot[i * Cfg::SP + n2];
  DFT<Cfg::N2, true, typename V2<R>::T>::run(v);
}

// I1 with the highest stored mode known at run time only (N / 3 < kmax < N / 2)
template <typename R, int N>
__device__ __forceinline__ void xr_i1_wide(const typename V2<R>::T* ra, const typename V2<R>::T* rb, int kmax, bool live,
                                           int j, const typename V2<R>::T* __restrict__ t1, typename V2<R>::T* slot) {
  using C = typename V2<R>::T;
  using Cfg = XRowCfg<R, N>;
  constexpr int N1 = Cfg::N1, N2 = Cfg::N2;
  C v[N1];
#pragma unroll
  for (int n1 = 0; n1 < N1; ++n1) {
    const int f = N2 * n1 + j;
    v[n1] = mk<C>(R(0), R(0));
    if (!live) continue;
    const int cls = crange(N2 * n1, N2, N, N / 3 + 1, N / 3);  // 0, 1: stored whatever kmax is
    if (cls == 0 || (2 * N2 * n1 < N && cls != 1 && f <= kmax)) v[n1] = xr_direct(ra, rb, f, n1 == 0 && j == 0);
    else if (cls == 1 || (2 * (N2 * n1 + N2) > N && f >= N - kmax)) v[n1] = xr_mirror(ra, rb, N - f);
  }
  DFT<N1, true, C>::run(v);
#pragma unroll
  for (int k1 = 1; k1 < N1; ++k1) {
    const C w = __ldg(t1 + k1 * N2 + j);
    v[k1] = cmul(v[k1], mk<C>(w.x, -w.y));
  }
#pragma unroll
  for (int k1 = 0; k1 < N1; ++k1) slot[k1 * Cfg::SP + j] = v[k1];
}

// F1 of lane i: v[n] = packed physical values at x = i + N1 n
template <typename R, int N>
__device__ __forceinline__ void xr_f1(typename V2<R>::T* v, int i, const typename V2<R>::T* __restrict__ t2,
                                      typename V2<R>::T* slot) {
  using Cfg = XRowCfg<R, N>;
  DFT<Cfg::N2, false, typename V2<R>::T>::run(v);
  slot[i] = v[0];
#pragma unroll
  for (int k = 1; k < Cfg::N2; ++k) slot[k * Cfg::SQ + i] = cmul(v[k], __ldg(t2 + k * Cfg::N1 + i));
}

// F2 of item k' in place: mode k = k' + N2 m goes to slot[k' SQ + m]; modes the
// truncation KMAX drops are not formed
template <typename R, int N, int KMAX>
__device__ __forceinline__ void xr_f2(typename V2<R>::T* slot, int kp) {
  using C = typename V2<R>::T;
  using Cfg = XRowCfg<R, N>;
  constexpr int N1 = Cfg::N1, N2 = Cfg::N2;
  constexpr int KNEG = 2 * KMAX == N ? KMAX - 1 : KMAX;
  C v[N1];
  C* p = slot + kp * Cfg::SQ;
#pragma unroll
  for (int m = 0; m < N1; ++m) v[m] = p[m];
  DFT<N1, false, C>::run(v);
#pragma unroll
  for (int m = 0; m < N1; ++m)
    if (crange(N2 * m, N2, N, KMAX + 1, KNEG) != 2) p[m] = v[m];
}

// place of mode k in a slot after F2
template <typename R, int N> __device__ __forceinline__ int xr_at(int k) {
  using Cfg = XRowCfg<R, N>;
  return (k % Cfg::N2) * Cfg::SQ + k / Cfg::N2;
}

// ---------------------------------------------------------------------------
// product sweep: c2r of the D velocity rows, u_i u_j * scale, r2c
// ---------------------------------------------------------------------------
// 3D pencils of a row pair (r, r + 1): slot 0 u1 + i u2 (r), slot 1 the same of
// r + 1, slot 2 u3(r) + i u3(r + 1); forward, one row at a time, in slots 0, 2,
// 3: (u1 u1, u2 u2), (u3 u3, u1 u2), (u2 u3, u3 u1).  2D: slots 0, 1 as above;
// forward (u1 u1, u2 u2) of each row and u1 u2 (r) + i u1 u2 (r + 1).
// FULL: all N / 3 + 1 modes are kept on the output.  WIDE: the rows hold up to
// N / 2 modes (the reduced grid of the DNS -> LES filter) and at most N / 5 + 1
// are kept, so that most of the last forward radix is never formed.
template <typename R, int N, int D, bool FULL, bool WIDE = false>
__global__ void __launch_bounds__(32 * XRowCfg<R, N>::wpc(D == 3 ? 4 : 3),
                                  XRowCfg<R, N>::minb(D == 3 ? 4 : 3, XRowCfg<R, N>::regs_ns))
k_xr_ns(const __grid_constant__ XArgs a, const typename V2<R>::T* __restrict__ t1, const typename V2<R>::T* __restrict__ t2) {
  using C = typename V2<R>::T;
  using Cfg = XRowCfg<R, N>;
  constexpr int N1 = Cfg::N1, N2 = Cfg::N2, W = Cfg::W, PS = Cfg::PS, KC = Cfg::KC;
  constexpr int NI = D == 3 ? 3 : 2;  // inverse pencils of a row pair
  constexpr int WPC = Cfg::wpc(D == 3 ? 4 : 3);
  constexpr int KO = WIDE ? N / 5 : KC;  // highest mode the forward side may keep
  const int K1i = WIDE ? a.K1in : KC + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  C* sm = reinterpret_cast<C*>(smem_raw + (threadIdx.x >> 5) * Cfg::slots(D == 3 ? 4 : 3));
  const int npair = int(a.nrows >> 1);  // N is even, so rows come in whole pairs
  const int rp0 = (int(blockIdx.x) * WPC + (threadIdx.x >> 5)) * W;
  if (rp0 >= npair) return;  // whole warps leave
  const C* in0 = static_cast<const C*>(a.in[0]);
  const C* in1 = static_cast<const C*>(a.in[1]);
  const C* in2 = static_cast<const C*>(a.in[D == 3 ? 2 : 1]);
#pragma unroll 1
  for (int it = lane; it < W * NI * N2; it += 32) {
    const int q = it / N2, j = it - q * N2, p = q / W, w = q - p * W;  // slot q: pencil p of row pair w
    const int row = 2 * (rp0 + w);
    const C* ra = (p < 2 ? in0 : in2) + (row + (p == 1)) * K1i;
    const C* rb = p < 2 ? in1 + (row + p) * K1i : in2 + (row + 1) * K1i;
    C* slot = sm + q * PS;
    if constexpr (WIDE) xr_i1_wide<R, N>(ra, rb, K1i - 1, rp0 + w < npair, j, t1, slot);
    else xr_i1<R, N, KC>(ra, rb, rp0 + w < npair, j, t1, slot);
  }
  __syncwarp();
  const int w = lane / N1, i = lane - w * N1;
  const bool act = w < W;
  const R hsc = R(0.5) * R(a.scale);
  const int K1o = FULL ? KC + 1 : a.K1out;
  const int ldo = a.ldo > 0 ? a.ldo : K1o;
  if constexpr (D == 3 && Cfg::IN_SLOTS) {
    // the lane's own points of slots 0..2 in place, then one forward pencil at a
    // time through slot 3
    C* own = sm + w * PS + i * Cfg::SP;
    if (act) {
#pragma unroll 1
      for (int p = 0; p < 3; ++p) {
        C v[N2];
        xr_i2<R, N>(sm + (p * W + w) * PS, i, v);
#pragma unroll
        for (int s = 0; s < N2; ++s) own[p * W * PS + s] = v[s];
      }
    }
#pragma unroll 1
    for (int r = 0; r < 2; ++r) {
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        if (act) {
          C v[N2];
#pragma unroll
          for (int s = 0; s < N2; ++s) {
            const C z = own[r * W * PS + s];
            const C y = own[2 * W * PS + s];
            const R u3 = r ? y.y : y.x;
            v[s] = b == 0 ? mk<C>(z.x * z.x, z.y * z.y) : b == 1 ? mk<C>(u3 * u3, z.x * z.y) : mk<C>(z.y * u3, u3 * z.x);
          }
          xr_f1<R, N>(v, i, t2, sm + (3 * W + w) * PS);
        }
        __syncwarp();
        for (int it = lane; it < W * N2; it += 32) xr_f2<R, N, KO>(sm + (3 * W + it / N2) * PS, it % N2);
        __syncwarp();
        for (int it = lane; it < W * K1o; it += 32) {
          const int ww = it / K1o, kx = it - ww * K1o;
          if (rp0 + ww >= npair) break;
          const int o = (2 * (rp0 + ww) + r) * ldo + kx;
          const C* z = sm + (3 * W + ww) * PS;
          const C x = z[xr_at<R, N>(kx)], y = z[xr_at<R, N>(kx == 0 ? 0 : N - kx)];
          static_cast<C*>(a.out[2 * b])[o] = mk<C>(hsc * (x.x + y.x), hsc * (x.y - y.y));
          static_cast<C*>(a.out[2 * b + 1])[o] = mk<C>(hsc * (x.y + y.y), hsc * (y.x - x.x));
        }
        __syncwarp();
      }
    }
  } else if constexpr (D == 3) {
    R u1[N2], u2[N2], u3[N2], u3b[N2];
    if (act) {
      C v[N2];
      xr_i2<R, N>(sm + (2 * W + w) * PS, i, v);
#pragma unroll
      for (int s = 0; s < N2; ++s) { u3[s] = v[s].x; u3b[s] = v[s].y; }
    }
#pragma unroll 1
    for (int r = 0; r < 2; ++r) {
      if (act) {
        C v[N2];
        xr_i2<R, N>(sm + (r * W + w) * PS, i, v);
#pragma unroll
        for (int s = 0; s < N2; ++s) { u1[s] = v[s].x; u2[s] = v[s].y; }
      }
      __syncwarp();
      if (act) {
        C v[N2];
#pragma unroll
        for (int s = 0; s < N2; ++s) v[s] = mk<C>(u1[s] * u1[s], u2[s] * u2[s]);
        xr_f1<R, N>(v, i, t2, sm + w * PS);
#pragma unroll
        for (int s = 0; s < N2; ++s) v[s] = mk<C>(u3[s] * u3[s], u1[s] * u2[s]);
        xr_f1<R, N>(v, i, t2, sm + (2 * W + w) * PS);
#pragma unroll
        for (int s = 0; s < N2; ++s) v[s] = mk<C>(u2[s] * u3[s], u3[s] * u1[s]);
        xr_f1<R, N>(v, i, t2, sm + (3 * W + w) * PS);
#pragma unroll
        for (int s = 0; s < N2; ++s) u3[s] = u3b[s];
      }
      __syncwarp();
#pragma unroll 1
      for (int it = lane; it < W * 3 * N2; it += 32) {
        const int q = it / N2, kp = it - q * N2;  // slot 0, 2, 3 of row pair q % W
        const int b = q / W;
        xr_f2<R, N, KO>(sm + ((b ? b + 1 : 0) * W + q - b * W) * PS, kp);
      }
      __syncwarp();
      for (int it = lane; it < W * K1o; it += 32) {
        const int ww = it / K1o, kx = it - ww * K1o;
        if (rp0 + ww >= npair) break;
        const int o = (2 * (rp0 + ww) + r) * ldo + kx;
        const int at = xr_at<R, N>(kx), an = xr_at<R, N>(kx == 0 ? 0 : N - kx);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          const C* z = sm + ((b ? b + 1 : 0) * W + ww) * PS;
          const C x = z[at], y = z[an];
          static_cast<C*>(a.out[2 * b])[o] = mk<C>(hsc * (x.x + y.x), hsc * (x.y - y.y));
          static_cast<C*>(a.out[2 * b + 1])[o] = mk<C>(hsc * (x.y + y.y), hsc * (y.x - x.x));
        }
      }
      __syncwarp();
    }
  } else {
    C v[N2], vx[N2], vb[N2];
    if (act) {
      xr_i2<R, N>(sm + w * PS, i, v);
      xr_i2<R, N>(sm + (W + w) * PS, i, vb);
    }
    __syncwarp();
    if (act) {
#pragma unroll
      for (int s = 0; s < N2; ++s) {
        vx[s] = mk<C>(v[s].x * v[s].y, vb[s].x * vb[s].y);
        v[s] = mk<C>(v[s].x * v[s].x, v[s].y * v[s].y);
        vb[s] = mk<C>(vb[s].x * vb[s].x, vb[s].y * vb[s].y);
      }
      xr_f1<R, N>(v, i, t2, sm + w * PS);
      xr_f1<R, N>(vb, i, t2, sm + (W + w) * PS);
      xr_f1<R, N>(vx, i, t2, sm + (2 * W + w) * PS);
    }
    __syncwarp();
#pragma unroll 1
    for (int it = lane; it < W * 3 * N2; it += 32) {
      const int q = it / N2, kp = it - q * N2;
      xr_f2<R, N, KC>(sm + q * PS, kp);
    }
    __syncwarp();
    for (int it = lane; it < W * K1o; it += 32) {
      const int ww = it / K1o, kx = it - ww * K1o;
      if (rp0 + ww >= npair) break;
      const int o = 2 * (rp0 + ww) * ldo + kx;
      const int at = xr_at<R, N>(kx), an = xr_at<R, N>(kx == 0 ? 0 : N - kx);
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const C* z = sm + (b * W + ww) * PS;
        const C x = z[at], y = z[an];
        const C xa = mk<C>(hsc * (x.x + y.x), hsc * (x.y - y.y)), xb = mk<C>(hsc * (x.y + y.y), hsc * (y.x - x.x));
        static_cast<C*>(a.out[b == 2 ? 2 : 0])[b == 1 ? o + ldo : o] = xa;
        static_cast<C*>(a.out[b == 2 ? 2 : 1])[b == 0 ? o : o + ldo] = xb;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// plain c2r / r2c of a batch: the rows of all fields are numbered one after
// another (rho = field * nrows + row) and packed in pairs (2q, 2q + 1), so a
// single field fills its pencils as well as a batch does
// ---------------------------------------------------------------------------
template <typename R, int N, int KMAX>
__global__ void __launch_bounds__(32 * XRowCfg<R, N>::wpc(3), XRowCfg<R, N>::minb(3, XRowCfg<R, N>::regs_plain))
k_xr_c2r(const __grid_constant__ XPlainArgs a, const typename V2<R>::T* __restrict__ t1) {
  using C = typename V2<R>::T;
  using Cfg = XRowCfg<R, N>;
  constexpr int N1 = Cfg::N1, N2 = Cfg::N2, PS = Cfg::PS, NP = 3 * Cfg::W, WPC = Cfg::wpc(3);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  C* sm = reinterpret_cast<C*>(smem_raw + (threadIdx.x >> 5) * Cfg::slots(3));
  const int nrow = int(a.nrows), npair = int(a.nrows >> 1) * a.ncomp;
  const int q0 = (int(blockIdx.x) * WPC + (threadIdx.x >> 5)) * NP;
  if (q0 >= npair) return;
#pragma unroll 1
  for (int it = lane; it < NP * N2; it += 32) {
    const int p = it / N2, j = it - p * N2, rho = 2 * (q0 + p);
    const int c = rho / nrow, row = rho - c * nrow;
    const bool live = q0 + p < npair;
    const C* ra = static_cast<const C*>(a.in[live ? c : 0]) + row * (KMAX + 1);
    xr_i1<R, N, KMAX>(ra, ra + KMAX + 1, live, j, t1, sm + p * PS);
  }
  __syncwarp();
  const R sc = R(a.scale);
#pragma unroll 1
  for (int it = lane; it < NP * N1; it += 32) {
    const int p = it / N1, i = it - p * N1, rho = 2 * (q0 + p);
    if (q0 + p >= npair) break;
    const int c = rho / nrow, row = rho - c * nrow;
    C v[N2];
    xr_i2<R, N>(sm + p * PS, i, v);
    R* o = static_cast<R*>(a.out[c]) + (long long)row * N + i;
#pragma unroll
    for (int k = 0; k < N2; ++k) { o[N1 * k] = v[k].x * sc; o[N + N1 * k] = v[k].y * sc; }
  }
}

template <typename R, int N, int KMAX>
__global__ void __launch_bounds__(32 * XRowCfg<R, N>::wpc(3), XRowCfg<R, N>::minb(3, XRowCfg<R, N>::regs_plain))
k_xr_r2c(const __grid_constant__ XPlainArgs a, const typename V2<R>::T* __restrict__ t2) {
  using C = typename V2<R>::T;
  using Cfg = XRowCfg<R, N>;
  constexpr int N1 = Cfg::N1, N2 = Cfg::N2, PS = Cfg::PS, NP = 3 * Cfg::W, WPC = Cfg::wpc(3), K1 = KMAX + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  C* sm = reinterpret_cast<C*>(smem_raw + (threadIdx.x >> 5) * Cfg::slots(3));
  const int nrow = int(a.nrows), npair = int(a.nrows >> 1) * a.ncomp;
  const int q0 = (int(blockIdx.x) * WPC + (threadIdx.x >> 5)) * NP;
  if (q0 >= npair) return;
  const R sc = R(a.scale);
#pragma unroll 1
  for (int it = lane; it < NP * N1; it += 32) {
    const int p = it / N1, i = it - p * N1, rho = 2 * (q0 + p);
    if (q0 + p >= npair) break;
    const int c = rho / nrow, row = rho - c * nrow;
    const R* x = static_cast<const R*>(a.in[c]) + (long long)row * N + i;
    C v[N2];
#pragma unroll
    for (int n = 0; n < N2; ++n) v[n] = mk<C>(__ldg(x + N1 * n) * sc, __ldg(x + N + N1 * n) * sc);
    xr_f1<R, N>(v, i, t2, sm + p * PS);
  }
  __syncwarp();
#pragma unroll 1
  for (int it = lane; it < NP * N2; it += 32) {
    const int p = it / N2, kp = it - p * N2;
    xr_f2<R, N, KMAX>(sm + p * PS, kp);
  }
  __syncwarp();
  for (int it = lane; it < NP * K1; it += 32) {
    const int p = it / K1, kx = it - p * K1, rho = 2 * (q0 + p);
    if (q0 + p >= npair) break;
    const int c = rho / nrow, row = rho - c * nrow;
    const C* z = sm + p * PS;
    const C x = z[xr_at<R, N>(kx)], y = z[xr_at<R, N>(kx == 0 ? 0 : N - kx)];
    C* o = static_cast<C*>(a.out[c]) + row * K1 + kx;
    o[0] = mk<C>(R(0.5) * (x.x + y.x), R(0.5) * (x.y - y.y));
    o[K1] = mk<C>(R(0.5) * (x.y + y.y), R(0.5) * (y.x - x.x));
  }
}

// ---------------------------------------------------------------------------
// closure sweep: c2r of NI fields, the closure's point function, r2c of the six
// stress components.  Pencil p of a row pair is field p's rows (r, r + 1), so a
// slot's place holds both rows' value of one point; the six stresses take the
// places of the first six fields.  Against c2r, point kernel and r2c it spares
// the write and the read of NI + 6 physical fields (128^3 FP32, six in six out:
// 66 us in three kernels).
// ---------------------------------------------------------------------------
template <typename R, int N, int NI>
__global__ void __launch_bounds__(32 * XRowCfg<R, N>::wpc(NI), XRowCfg<R, N>::minb(NI, XRowCfg<R, N>::regs_plain))
k_xr_point(const __grid_constant__ XPointArgs a, const typename V2<R>::T* __restrict__ t1,
           const typename V2<R>::T* __restrict__ t2) {
  using C = typename V2<R>::T;
  using Cfg = XRowCfg<R, N>;
  constexpr int N1 = Cfg::N1, N2 = Cfg::N2, W = Cfg::W, PS = Cfg::PS, KC = Cfg::KC, K1 = KC + 1, WPC = Cfg::wpc(NI);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  C* sm = reinterpret_cast<C*>(smem_raw + (threadIdx.x >> 5) * Cfg::slots(NI));
  const int npair = int(a.nrows >> 1);
  const int rp0 = (int(blockIdx.x) * WPC + (threadIdx.x >> 5)) * W;
  if (rp0 >= npair) return;
#pragma unroll 1
  for (int it = lane; it < W * NI * N2; it += 32) {
    const int q = it / N2, j = it - q * N2, p = q / W, w = q - p * W;  // slot q: field p of row pair w
    const C* ra = static_cast<const C*>(a.in[p]) + 2 * (rp0 + w) * K1;
    xr_i1<R, N, KC>(ra, ra + K1, rp0 + w < npair, j, t1, sm + q * PS);
  }
  __syncwarp();
  const int w = lane / N1, i = lane - w * N1;
  const bool act = w < W;
  C* own = sm + w * PS + i * Cfg::SP;  // this lane's points of field p at own[p W PS + s]
  if (act) {
#pragma unroll 1
    for (int p = 0; p < NI; ++p) {
      C v[N2];
      xr_i2<R, N>(sm + (p * W + w) * PS, i, v);
#pragma unroll
      for (int s = 0; s < N2; ++s) own[p * W * PS + s] = v[s];
    }
    const R d2 = R(a.delta * a.delta), p0 = R(a.p0);
#pragma unroll 1
    for (int s = 0; s < N2; ++s) {
      C z[NI];
#pragma unroll
      for (int p = 0; p < NI; ++p) z[p] = own[p * W * PS + s];
      if constexpr (NI == 6) {
        R x[6], y[6];
#pragma unroll
        for (int p = 0; p < 6; ++p) { x[p] = z[p].x; y[p] = z[p].y; }
        const R nx = smag_viscosity<R, 3>(d2, x), ny = smag_viscosity<R, 3>(d2, y);
#pragma unroll
        for (int p = 0; p < 6; ++p) own[p * W * PS + s] = mk<C>(-R(2) * nx * x[p], -R(2) * ny * y[p]);
      } else {
        R G[2][3][3], t[2][3][3];
#pragma unroll
        for (int p = 0; p < 9; ++p) { G[0][p % 3][p / 3] = z[p].x; G[1][p % 3][p / 3] = z[p].y; }
        closure_point<R, 3>(a.kind, d2, p0, G[0], t[0]);
        closure_point<R, 3>(a.kind, d2, p0, G[1], t[1]);
        constexpr int PI[6] = {0, 1, 2, 0, 1, 2}, PJ[6] = {0, 1, 2, 1, 2, 0};
#pragma unroll
        for (int p = 0; p < 6; ++p) own[p * W * PS + s] = mk<C>(t[0][PI[p]][PJ[p]], t[1][PI[p]][PJ[p]]);
      }
    }
  }
#pragma unroll 1
  for (int p = 0; p < 6; ++p) {
    C v[N2];
    if (act) {
#pragma unroll
      for (int s = 0; s < N2; ++s) v[s] = own[p * W * PS + s];
    }
    __syncwarp();
    if (act) xr_f1<R, N>(v, i, t2, sm + (p * W + w) * PS);
  }
  __syncwarp();
#pragma unroll 1
  for (int it = lane; it < W * 6 * N2; it += 32) {
    const int q = it / N2, kp = it - q * N2;
    xr_f2<R, N, KC>(sm + q * PS, kp);
  }
  __syncwarp();
  const R hsc = R(0.5) * R(a.scale);
  for (int it = lane; it < W * K1; it += 32) {
    const int ww = it / K1, kx = it - ww * K1;
    if (rp0 + ww >= npair) break;
    const int o = 2 * (rp0 + ww) * K1 + kx;
    const int at = xr_at<R, N>(kx), an = xr_at<R, N>(kx == 0 ? 0 : N - kx);
#pragma unroll
    for (int p = 0; p < 6; ++p) {
      const C* z = sm + (p * W + ww) * PS;
      const C x = z[at], y = z[an];
      static_cast<C*>(a.out[p])[o] = mk<C>(hsc * (x.x + y.x), hsc * (x.y - y.y));
      static_cast<C*>(a.out[p])[o + K1] = mk<C>(hsc * (x.y + y.y), hsc * (y.x - x.x));
    }
  }
}

// ---------------------------------------------------------------------------
// max over the physical points of |u|^2 (FP64) of D fields of rows
// (propose_timestep, src/solver.jl:931-947); *out is the bit pattern of the
// largest value so far (non-negative doubles order like their bits)
// ---------------------------------------------------------------------------
template <typename R, int N, int D>
__global__ void __launch_bounds__(32 * XRowCfg<R, N>::wpc(3), XRowCfg<R, N>::minb(3, XRowCfg<R, N>::regs_ns))
k_xr_vmax(const __grid_constant__ XPlainArgs a, const typename V2<R>::T* __restrict__ t1, unsigned long long* out) {
  using C = typename V2<R>::T;
  using Cfg = XRowCfg<R, N>;
  constexpr int N1 = Cfg::N1, N2 = Cfg::N2, W = Cfg::W, PS = Cfg::PS, KC = Cfg::KC, WPC = Cfg::wpc(3);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31;
  C* sm = reinterpret_cast<C*>(smem_raw + (threadIdx.x >> 5) * Cfg::slots(3));
  const int npair = int(a.nrows >> 1);
  const int rp0 = (int(blockIdx.x) * WPC + (threadIdx.x >> 5)) * W;
  if (rp0 >= npair) return;
  const C* in0 = static_cast<const C*>(a.in[0]);
  const C* in1 = static_cast<const C*>(a.in[1]);
  const C* in2 = static_cast<const C*>(a.in[D == 3 ? 2 : 1]);
#pragma unroll 1
  for (int it = lane; it < W * D * N2; it += 32) {
    const int q = it / N2, j = it - q * N2, p = q / W, w = q - p * W;
    const int row = 2 * (rp0 + w);
    const C* ra = (p < 2 ? in0 : in2) + (row + (p == 1)) * (KC + 1);
    const C* rb = p < 2 ? in1 + (row + p) * (KC + 1) : in2 + (row + 1) * (KC + 1);
    xr_i1<R, N, KC>(ra, rb, rp0 + w < npair, j, t1, sm + q * PS);
  }
  __syncwarp();
  const int w = lane / N1, i = lane - w * N1;
  double m = 0;
  if (w < W && rp0 + w < npair) {
    double s0[N2], s1[N2];  // |u|^2 of the two rows
    C v[N2];
#pragma unroll
    for (int s = 0; s < N2; ++s) s0[s] = s1[s] = 0.0;
#pragma unroll
    for (int p = 0; p < D; ++p) {
      xr_i2<R, N>(sm + (p * W + w) * PS, i, v);
#pragma unroll
      for (int s = 0; s < N2; ++s) {
        const double x = v[s].x, y = v[s].y;
        if (p == 0) s0[s] = x * x + y * y;
        else if (p == 1) s1[s] = x * x + y * y;
        else { s0[s] += x * x; s1[s] += y * y; }
      }
    }
#pragma unroll
    for (int s = 0; s < N2; ++s) {
      m = s0[s] > m ? s0[s] : m;
      m = s1[s] > m ? s1[s] : m;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double q = __shfl_down_sync(0xffffffffu, m, o);
    m = q > m ? q : m;
  }
  if (lane == 0) atomicMax(out, (unsigned long long)__double_as_longlong(m));
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
template <typename F> static void xr_smem(F* f, size_t bytes) {
  if (bytes > 48 * 1024) cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
}

template <typename R, int N> void XRow<R, N>::init() {
  using Cfg = XRowCfg<R, N>;
  constexpr size_t s3 = Cfg::wpc(3) * Cfg::slots(3), s4 = Cfg::wpc(4) * Cfg::slots(4);
  xr_smem(k_xr_ns<R, N, 3, true>, s4);
  xr_smem(k_xr_ns<R, N, 3, false>, s4);
  xr_smem(k_xr_ns<R, N, 3, false, true>, s4);
  xr_smem(k_xr_ns<R, N, 2, true>, s3);
  xr_smem(k_xr_ns<R, N, 2, false>, s3);
  xr_smem(k_xr_c2r<R, N, N / 3>, s3);
  xr_smem(k_xr_c2r<R, N, N / 2>, s3);
  xr_smem(k_xr_r2c<R, N, N / 3>, s3);
  xr_smem(k_xr_r2c<R, N, N / 2>, s3);
  xr_smem(k_xr_point<R, N, 6>, Cfg::wpc(6) * Cfg::slots(6));
  xr_smem(k_xr_point<R, N, 9>, Cfg::wpc(9) * Cfg::slots(9));
  xr_smem(k_xr_vmax<R, N, 2>, s3);
  xr_smem(k_xr_vmax<R, N, 3>, s3);
}

// warps needed for `items` of `per` a warp, in CTAs of wpc warps
static inline unsigned xr_grid(long long items, int per, int wpc) {
  return unsigned((items + (long long)per * wpc - 1) / ((long long)per * wpc));
}

template <typename R, int N> void XRow<R, N>::ns(const XArgs& a, const void* tx, cudaStream_t st) {
  using C = typename V2<R>::T;
  using Cfg = XRowCfg<R, N>;
  const C* t1 = static_cast<const C*>(tx);
  const C* t2 = t1 + N;
  if (a.D == 2) {
    constexpr int wpc = Cfg::wpc(3);
    const unsigned nb = xr_grid(a.nrows / 2, Cfg::W, wpc);
    if (a.K1out == N / 3 + 1) k_xr_ns<R, N, 2, true><<<nb, 32 * wpc, wpc * Cfg::slots(3), st>>>(a, t1, t2);
    else k_xr_ns<R, N, 2, false><<<nb, 32 * wpc, wpc * Cfg::slots(3), st>>>(a, t1, t2);
    return;
  }
  constexpr int wpc = Cfg::wpc(4);
  const unsigned nb = xr_grid(a.nrows / 2, Cfg::W, wpc);
  if (a.K1in != N / 3 + 1) k_xr_ns<R, N, 3, false, true><<<nb, 32 * wpc, wpc * Cfg::slots(4), st>>>(a, t1, t2);
  else if (a.K1out == N / 3 + 1) k_xr_ns<R, N, 3, true><<<nb, 32 * wpc, wpc * Cfg::slots(4), st>>>(a, t1, t2);
  else k_xr_ns<R, N, 3, false><<<nb, 32 * wpc, wpc * Cfg::slots(4), st>>>(a, t1, t2);
}

template <typename R, int N> void XRow<R, N>::c2r(const XPlainArgs& a, const void* tx, cudaStream_t st) {
  using C = typename V2<R>::T;
  using Cfg = XRowCfg<R, N>;
  constexpr int wpc = Cfg::wpc(3);
  const C* t1 = static_cast<const C*>(tx);
  const unsigned nb = xr_grid(a.nrows / 2 * a.ncomp, 3 * Cfg::W, wpc);
  if (a.K1 == N / 2 + 1) k_xr_c2r<R, N, N / 2><<<nb, 32 * wpc, wpc * Cfg::slots(3), st>>>(a, t1);
  else k_xr_c2r<R, N, N / 3><<<nb, 32 * wpc, wpc * Cfg::slots(3), st>>>(a, t1);
}

template <typename R, int N> void XRow<R, N>::r2c(const XPlainArgs& a, const void* tx, cudaStream_t st) {
  using C = typename V2<R>::T;
  using Cfg = XRowCfg<R, N>;
  constexpr int wpc = Cfg::wpc(3);
  const C* t2 = static_cast<const C*>(tx) + N;
  const unsigned nb = xr_grid(a.nrows / 2 * a.ncomp, 3 * Cfg::W, wpc);
  if (a.K1 == N / 2 + 1) k_xr_r2c<R, N, N / 2><<<nb, 32 * wpc, wpc * Cfg::slots(3), st>>>(a, t2);
  else k_xr_r2c<R, N, N / 3><<<nb, 32 * wpc, wpc * Cfg::slots(3), st>>>(a, t2);
}

template <typename R, int N> void XRow<R, N>::point(const XPointArgs& a, const void* tx, cudaStream_t st) {
  using C = typename V2<R>::T;
  using Cfg = XRowCfg<R, N>;
  const C* t1 = static_cast<const C*>(tx);
  if (a.nin == 6) {
    constexpr int wpc = Cfg::wpc(6);
    k_xr_point<R, N, 6><<<xr_grid(a.nrows / 2, Cfg::W, wpc), 32 * wpc, wpc * Cfg::slots(6), st>>>(a, t1, t1 + N);
  } else {
    constexpr int wpc = Cfg::wpc(9);
    k_xr_point<R, N, 9><<<xr_grid(a.nrows / 2, Cfg::W, wpc), 32 * wpc, wpc * Cfg::slots(9), st>>>(a, t1, t1 + N);
  }
}

template <typename R, int N>
void XRow<R, N>::vmax(const XPlainArgs& a, const void* tx, unsigned long long* out, cudaStream_t st) {
  using C = typename V2<R>::T;
  using Cfg = XRowCfg<R, N>;
  constexpr int wpc = Cfg::wpc(3);
  const C* t1 = static_cast<const C*>(tx);
  const unsigned nb = xr_grid(a.nrows / 2, Cfg::W, wpc);
  if (a.ncomp == 2) k_xr_vmax<R, N, 2><<<nb, 32 * wpc, wpc * Cfg::slots(3), st>>>(a, t1, out);
  else k_xr_vmax<R, N, 3><<<nb, 32 * wpc, wpc * Cfg::slots(3), st>>>(a, t1, out);
}

}  // namespace sc
