// Weight and bias gradients of the closure network's convolutions on tcgen05
// tensor cores (sc_wgrad.cu).
#pragma once
#include "sc_cnn.h"

namespace sc {

struct WgradArgs {
  const __nv_bfloat16* g;    // output gradient, channels-last [n^3][COP]: BF16 (high parts)
  const __nv_bfloat16* glo;  // split precision: BF16 low parts
  const void* a;             // layer input [n^3][CP]: BF16, or FP16 high parts in split precision
  const void* alo;           // split precision: FP16 low parts
  int cin, cout;             // the layer's own channels (<= CP, COP)
  double* gw;                // += [cout][cin][27]
  double* gb;                // += [cout]
  int* err;                  // set when a bounded wait ran out
  int nsm;
  long long wait_limit;
};

void wgrad_init();
// n = 64 or 128; (CP, COP) = (16, 32), (32, 32) or (32, 16)
void launch_wgrad(int n, int cp, int cop, bool split, const WgradArgs& a, cudaStream_t st);

}  // namespace sc
