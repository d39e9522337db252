// Weight and bias gradients of the closure network's 3x3x3 convolutions on the
// 5th-generation tensor cores:
//   gw[co][ci][t] += sum_v g[v][co] a[v + off(t)][ci],  gb[co] += sum_v g[v][co].
//
// Per tap this is a GEMM whose contraction runs over the voxels, with both
// operands channels-last, so both enter the MMA MN-major: a staged plane holds 8
// channels of a row of voxels at 16 bytes a voxel, K = 16 voxels is two groups
// of 8 consecutive 16-byte units, and the x shift of a tap is a 16-byte offset
// of the descriptor.  One MMA covers the three y shifts at once (N = 3 CP: the
// planes of three consecutive input rows are consecutive in shared memory), the
// three x shifts are three accumulators of 3 CP columns, and the z shift is the
// CTA's own, so a CTA holds 9 taps in tensor memory.
//
// Precision: the operands are split into BF16 parts whose products are exact in
// FP32.  Split-precision gradients g are two BF16 parts already; they are stacked
// along M (rows 0.. COP-1 high, COP.. 2 COP-1 low, added at the end).  The layer
// inputs, FP16 high and low parts of 22 bits together, are staged as three BF16
// parts (24 bits), accumulated by three MMAs.  So every product of the two sums
// is formed, as by the FP32 kernel this replaces.  M is 128 whatever the number
// of valid rows; the other rows multiply whatever follows in shared memory and
// are never read.
//
// The tensor core truncates its FP32 accumulations: over a CTA's thousand of them
// the gradient was off by 1.7e-5 where the FP32 kernel's was off by 4.2e-6.  So
// every half block starts from zero (8 accumulations of a size with the sum) and
// eight warps add its result to FP32 sums in registers.  What truncation has then
// taken from a result is within 20 % one part in 2^23 of it, whatever the data
// (white 1.0e-7 to 1.1e-7, smooth 1.0e-7 to 1.2e-7; all terms of one sign 1.6e-7),
// so the addition gives it back as an FMA with 1 + 2^-23.  Against FP64, 64^3,
// 32 -> 32, split, white | smooth data: read out once a block 2.7e-7 | 2.3e-7, the
// FP32 kernel 4.1e-7 | 2.4e-8.
//
// A block is 4 output rows of 64 voxels: 4 g rows and 6 input rows, staged by
// seven warps in one of two buffers while the MMA thread works on the other.
// What bounds it: the MMAs, about 88 cycles each whatever their N, and M half
// used.  64^3, 32 -> 32, split: 160 us read out once a block, 165 us twice, 963 us
// on CUDA cores.
#include <cuda_fp16.h>

#include "sc_tcgen05.cuh"
#include "sc_wgrad.h"

namespace sc {

namespace {
// 16 warps (128 registers a thread): by pairs, two that read out (tensor-memory
// lane quadrants 0 and 1, which hold the valid rows) and two that stage, except
// that warp 2 issues the MMAs
constexpr int kThreads = 512, kStage = 7 * 32, kMmaWarp = 2;
constexpr int TX = 64, YB = 4;         // voxels of a row tile, output rows of a block
constexpr int SB = 2, NSB = YB / SB;   // output rows, read-outs of a block
constexpr int PLANE = (TX + 2) * 16;   // bytes of 8 channels of a row with its x halo
// 16-byte x 8 stores of consecutive threads fall on distinct banks: PLANE = 32 (mod 128)
static_assert(PLANE % 128 == 32, "plane stride");

template <int CP, int COP, bool SPLIT> struct WgCfg {
  static constexpr int CI = CP / 8, CO = COP / 8;   // 16-byte channel chunks
  static constexpr int PA = SPLIT ? 3 : 1, PG = SPLIT ? 2 : 1;
  static constexpr int GPL = PG * CO;               // planes of one g row
  static constexpr int GB = YB * GPL * PLANE;
  static constexpr int AB = PA * (YB + 2) * CI * PLANE;
  static constexpr int BUF = GB + AB;
  static constexpr int NN = 3 * CP;                 // MMA N: three y shifts
  static constexpr int NCOL = 3 * NN;               // accumulator columns: three x shifts
  static constexpr int ROWS = PG * COP;             // valid accumulator rows (<= 64)
  static constexpr int RED = ROWS * (NCOL + 1) * 4;
  static constexpr int BODY = 2 * BUF > RED ? 2 * BUF : RED;
  static constexpr int SMEM = (BODY + 127) / 128 * 128 + 128;
  // the 16 planes of an A operand reach past the g rows into the input rows, no further
  static_assert((YB - 1) * GPL + 16 <= BUF / PLANE && SMEM <= 232448 && NCOL <= 512 && ROWS <= 64, "wgrad layout");
};

template <int NOUT> __host__ __device__ constexpr uint32_t mn_idesc() {
  // D f32; A and B bf16, both MN-major (bits 15, 16); N >> 3 at bit 17; M = 128
  return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | (uint32_t(NOUT >> 3) << 17) | (8u << 24);
}

__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  return uint32_t(__bfloat16_as_ushort(lo)) | (uint32_t(__bfloat16_as_ushort(hi)) << 16);
}
}  // namespace

template <int KN, int CP, int COP, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 1) k_wgrad_tc(const WgradArgs p) {
  using Cfg = WgCfg<CP, COP, SPLIT>;
  constexpr int CI = Cfg::CI, CO = Cfg::CO, PA = Cfg::PA, GPL = Cfg::GPL;
  extern __shared__ __align__(128) unsigned char sm[];
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + Cfg::SMEM - 128);  // [2] staged by all staging threads
  uint64_t* done = full + 2;                                            // [2] MMAs of the buffer's block complete
  uint64_t* summed = done + 2;                                          // MMAs of SB rows complete
  uint64_t* drained = summed + 1;                                       // accumulators of SB rows read out
  uint32_t* tslot = reinterpret_cast<uint32_t*>(drained + 1);
  int* abort_flag = reinterpret_cast<int*>(tslot + 1);
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const bool reader = !(warp & 2), stager = (warp & 2) && warp != kMmaWarp;
  const int sid = ((warp >> 2) * 2 + (warp & 1) - 1) * 32 + lane;  // rank among the stagers
  const int dzi = blockIdx.x % 3;  // z shift dzi - 1
  const int nct = (int(gridDim.x) - dzi + 2) / 3, cta = blockIdx.x / 3;
  constexpr int NBLK = KN * (KN / YB) * (KN / TX);
  const int b0 = int((long long)NBLK * cta / nct), b1 = int((long long)NBLK * (cta + 1) / nct);
  if (tid == 0) {
    for (int q = 0; q < 2; ++q) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(full + q)), "r"(kStage));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(done + q)));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(summed)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 8;" ::"r"(smem_u32(drained)));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    *abort_flag = 0;
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tslot;
  // bounded wait; gives up too once another thread's wait ran out
  auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
    for (long long it = 0; it < p.wait_limit; ++it) {
      if (mbar_wait(bar, parity, 1)) return true;
      if ((it & 15) == 15 && *reinterpret_cast<volatile int*>(abort_flag)) return false;
    }
    *reinterpret_cast<volatile int*>(abort_flag) = 1;
    return false;
  };
  bool ok = true;
  int last = -1;  // MMA thread: last committed block
  float gsum[8] = {};
  constexpr int NCOL = Cfg::NCOL, NCH = (NCOL / 16 + 3) / 4;  // 16-column chunks of a reader warp
  float acc[NCH][16] = {};
  if (stager) {
    static_assert(kStage % CO == 0, "a staging thread keeps its channel chunk of g");
    const int gc = sid % CO;
    for (int b = b0; b < b1 && ok; ++b) {
      const int i = b - b0, buf = i & 1;
      unsigned char* sg = sm + buf * Cfg::BUF;
      unsigned char* sa = sg + Cfg::GB;
      const int x0 = (b % (KN / TX)) * TX, y0 = (b / (KN / TX)) % (KN / YB) * YB, z = b / ((KN / TX) * (KN / YB));
      // block i - 2 has left this buffer
      if (i >= 2) ok = wait(done + buf, uint32_t((i >> 1) - 1) & 1u);
      if (!ok) break;
      const long long grow = ((long long)z * KN + y0) * KN + x0;
#pragma unroll 2
      for (int u = sid; u < YB * TX * CO; u += kStage) {
        const int v = (u / CO) % TX, r = u / (CO * TX);
        const long long q = (grow + (long long)r * KN + v) * COP + gc * 8;
        const uint4 h = __ldg(reinterpret_cast<const uint4*>(p.g + q));
        unsigned char* d = sg + (r * GPL + gc) * PLANE + v * 16;
        *reinterpret_cast<uint4*>(d) = h;
        uint4 l = make_uint4(0, 0, 0, 0);
        if (SPLIT) {
          l = __ldg(reinterpret_cast<const uint4*>(p.glo + q));
          *reinterpret_cast<uint4*>(d + CO * PLANE) = l;
        }
        if (dzi == 1) {
          const uint32_t hw[4] = {h.x, h.y, h.z, h.w}, lw[4] = {l.x, l.y, l.z, l.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            gsum[2 * e] += __uint_as_float(hw[e] << 16) + __uint_as_float(lw[e] << 16);
            gsum[2 * e + 1] += __uint_as_float(hw[e] & 0xffff0000u) + __uint_as_float(lw[e] & 0xffff0000u);
          }
        }
      }
      const int zz = (z + dzi - 1 + KN) % KN;
#pragma unroll 2
      for (int u = sid; u < (YB + 2) * (TX + 2) * CI; u += kStage) {
        const int c = u % CI, v = (u / CI) % (TX + 2), r = u / (CI * (TX + 2));
        const int yy = (y0 + r - 1 + KN) % KN, xx = (x0 + v - 1 + KN) % KN;
        const long long q = (((long long)zz * KN + yy) * KN + xx) * CP + c * 8;
        unsigned char* d = sa + (r * CI + c) * PLANE + v * 16;
        const uint4 h = __ldg(reinterpret_cast<const uint4*>(static_cast<const unsigned short*>(p.a) + q));
        if (!SPLIT) {
          *reinterpret_cast<uint4*>(d) = h;
        } else {
          const uint4 l = __ldg(reinterpret_cast<const uint4*>(static_cast<const unsigned short*>(p.alo) + q));
          const uint32_t hw[4] = {h.x, h.y, h.z, h.w}, lw[4] = {l.x, l.y, l.z, l.w};
          uint32_t o[3][4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 fh = __half22float2(*reinterpret_cast<const __half2*>(&hw[e]));
            const float2 fl = __half22float2(*reinterpret_cast<const __half2*>(&lw[e]));
            float x = fh.x + fl.x, y = fh.y + fl.y;  // exact: 22 bits
#pragma unroll
            for (int k = 0; k < 3; ++k) {
              const __nv_bfloat16 bx = __float2bfloat16_rn(x), by = __float2bfloat16_rn(y);
              o[k][e] = pack2(bx, by);
              x -= __bfloat162float(bx);
              y -= __bfloat162float(by);
            }
          }
#pragma unroll
          for (int k = 0; k < 3; ++k)
            *reinterpret_cast<uint4*>(d + k * (YB + 2) * CI * PLANE) = make_uint4(o[k][0], o[k][1], o[k][2], o[k][3]);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(full + buf)) : "memory");
    }
  } else if (reader) {
    const uint32_t ta = tmem + (uint32_t(32 * (warp & 1)) << 16);
    for (int q = 0; q < (b1 - b0) * NSB; ++q) {
      ok = __all_sync(0xffffffffu, wait(summed, uint32_t(q) & 1u));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
      if (32 * (warp & 1) < Cfg::ROWS) {
#pragma unroll
        for (int c = 0; c < NCH; ++c) {
          const int c0 = ((warp >> 2) + 4 * c) * 16;
          if (c0 < NCOL) {
            float v[16];
            tmem_ld<16>(ta + uint32_t(c0), v);
#pragma unroll
            for (int e = 0; e < 16; ++e) acc[c][e] = fmaf(v[e], 1.00000011920928955f, acc[c][e]);  // 1 + 2^-23
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(drained)) : "memory");
    }
  } else if (lane == 0) {
    constexpr uint32_t IDESC = mn_idesc<Cfg::NN>();
    const uint64_t D0 = make_desc(smem_u32(sm), 128, PLANE);
    for (int b = b0; b < b1 && ok; ++b) {
      const int i = b - b0, buf = i & 1;
      ok = wait(full + buf, uint32_t(i >> 1) & 1u);
      if (!ok) break;
      const uint32_t og = uint32_t(buf * Cfg::BUF) >> 4, oa = og + uint32_t(Cfg::GB >> 4);
#pragma unroll 1
      for (int h = 0; h < NSB; ++h) {
        const int q = i * NSB + h;
        if (q > 0 && !(ok = wait(drained, uint32_t(q - 1) & 1u))) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        // smallest part first: the high part's accumulations are then the only
        // ones that truncate at the size of the sum
#pragma unroll 1
        for (int k = PA - 1; k >= 0; --k)
#pragma unroll 1
          for (int yk = 0; yk < SB * (TX / 16); ++yk) {
            const int yl = h * SB + yk / (TX / 16), ks = yk % (TX / 16);
            const uint64_t da = D0 + og + uint32_t(yl * GPL * (PLANE >> 4) + ks * 16);
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
              const uint64_t db = D0 + oa + uint32_t((k * (YB + 2) + yl) * CI * (PLANE >> 4) + ks * 16 + dx);
              const uint32_t add = (yk > 0 || k < PA - 1) ? 1u : 0u;
              asm volatile(
                  "{\n\t.reg .pred p;\n\t"
                  "setp.ne.b32 p, %4, 0;\n\t"
                  "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                  :
                  : "r"(tmem + uint32_t(dx * Cfg::NN)), "l"(da), "l"(db), "r"(IDESC), "r"(add));
            }
          }
        mma_commit(summed);
      }
      // also after a wait that ran out: the exit waits for what was issued
      mma_commit(done + buf);
      last = b;
    }
    // all MMAs complete in order: the last commit covers every earlier one (on a
    // timeout with the default bound, before tensor and shared memory go)
    if (last >= 0) {
      const int i = last - b0;
      if (!mbar_wait(done + (i & 1), uint32_t(i >> 1) & 1u, ok ? p.wait_limit : kDefaultWaitLimit)) ok = false;
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  ok = __syncthreads_and(ok) != 0;
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (!ok) {
    if (tid == 0) atomicExch(p.err, 1);
    // the MMA thread may have given up on its last wait only just now
    if (last >= 0) {
      const int i = last - b0;
      mbar_wait(done + (i & 1), uint32_t(i >> 1) & 1u, kDefaultWaitLimit);
    }
  } else if (b1 > b0) {
    // sums -> shared memory [row][column], then high + low rows into the gradient
    constexpr int ROWS = Cfg::ROWS;
    float* red = reinterpret_cast<float*>(sm);
    const int row = 32 * (warp & 1) + lane;
    if (reader && row < ROWS) {
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        const int c0 = ((warp >> 2) + 4 * c) * 16;
        if (c0 < NCOL) {
#pragma unroll
          for (int e = 0; e < 16; ++e) red[row * (NCOL + 1) + c0 + e] = acc[c][e];
        }
      }
    }
    __syncthreads();
    // entry (co, ci, dy, dx): column dx NN + dy CP + ci
    for (int o = tid; o < p.cout * p.cin * 9; o += kThreads) {
      const int t9 = o % 9, ci = (o / 9) % p.cin, co = o / (9 * p.cin);
      const int col = (t9 % 3) * Cfg::NN + (t9 / 3) * CP + ci;
      double s = double(red[co * (NCOL + 1) + col]);
      if (SPLIT) s += double(red[(COP + co) * (NCOL + 1) + col]);
      atomicAdd(&p.gw[((long long)co * p.cin + ci) * 27 + dzi * 9 + t9], s);
    }
    if (dzi == 1) {  // bias: the staging threads' channel sums
      __syncthreads();
      if (stager) {
#pragma unroll
        for (int e = 0; e < 8; ++e) red[(sid / CO) * COP + (sid % CO) * 8 + e] = gsum[e];
      }
      __syncthreads();
      if (tid < p.cout) {
        double s = 0;
        for (int q = 0; q < kStage / CO; ++q) s += double(red[q * COP + tid]);
        atomicAdd(&p.gb[tid], s);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == kMmaWarp) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

template <int KN, int CP, int COP, bool SPLIT> static void wg_init() {
  cudaFuncSetAttribute(k_wgrad_tc<KN, CP, COP, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       WgCfg<CP, COP, SPLIT>::SMEM);
}
template <int KN> static void wg_init_n() {
  wg_init<KN, 16, 32, false>(); wg_init<KN, 32, 32, false>(); wg_init<KN, 32, 16, false>();
  wg_init<KN, 16, 32, true>(); wg_init<KN, 32, 32, true>(); wg_init<KN, 32, 16, true>();
}
void wgrad_init() {
  wg_init_n<64>();
  wg_init_n<128>();
}

template <int KN, int CP, int COP> static void wg_launch(bool split, const WgradArgs& a, cudaStream_t st) {
  const int grid = a.nsm >= 3 ? a.nsm : 148;
  if (split) k_wgrad_tc<KN, CP, COP, true><<<grid, kThreads, WgCfg<CP, COP, true>::SMEM, st>>>(a);
  else k_wgrad_tc<KN, CP, COP, false><<<grid, kThreads, WgCfg<CP, COP, false>::SMEM, st>>>(a);
}
template <int KN> static void wg_launch_n(int cp, int cop, bool split, const WgradArgs& a, cudaStream_t st) {
  if (cp == 16) wg_launch<KN, 16, 32>(split, a, st);
  else if (cop == 16) wg_launch<KN, 32, 16>(split, a, st);
  else wg_launch<KN, 32, 32>(split, a, st);
}
void launch_wgrad(int n, int cp, int cop, bool split, const WgradArgs& a, cudaStream_t st) {
  if (n == 64) wg_launch_n<64>(cp, cop, split, a, st);
  else wg_launch_n<128>(cp, cop, split, a, st);
}

}  // namespace sc
