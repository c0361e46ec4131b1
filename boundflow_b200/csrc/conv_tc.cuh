// Problem description of the tensor-core ReLU + transposed convolution (conv_tc.cu).
#pragma once
#include "kernels.cuh"

namespace bf {

struct ConvTcProblem {
  const float* A;                                // [M, Co, WH, WW] coefficients w.r.t. the ReLU output (or the conv output without slopes)
  const float *dpos, *dneg, *epos, *eneg, *add;  // [D, Co, WH, WW]; dpos null: no ReLU
  const float* bias;                             // [Co] or null
  const float* W;                                // [Co, Ci, kh, kw]
  float* out;                                    // [M, Ci, Hi, Wi]
  float* partial;                                // [M, slots] sums of a * intercept + lam * bias, or null
  int* status;                                   // device word, set non-zero when a wait expired (null: the NaN rows are the only sign)
  int M, S, Co, Ci, WH, WW, Hi, Wi, kh, kw, sh, sw, ph, pw;
};

// false: this geometry stays on the FP32 kernels.  slots: partial sums per row, tiles: 128-position tiles of the problem,
// us: the time the kernel is expected to take.
bool conv_tc_supports(const ConvTcProblem& c, int* slots, int* tiles, double* us);
int launch_conv_tc(const ConvTcProblem& c, cudaStream_t stream);

}  // namespace bf
