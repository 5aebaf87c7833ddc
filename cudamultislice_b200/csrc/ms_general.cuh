// ms_general.cuh -- conventional slice passes for line lengths that are no
// power of two.
//
// The same two passes per slice as ms_slice.cuh (rows: [IFFT] -> x exp(i sigma V)
// -> [FFT]; columns of the band: FFT -> x P/N -> IFFT) with mixed-radix Stockham
// transforms of a line in shared memory, for lengths 2..4096 whose prime
// factors are at most 13.  Other lengths stay on the plain path (cuFFT and one
// kernel per operation).
#pragma once
#include <cuda_runtime.h>

#include "ms_common.cuh"

namespace ms {

// Radix passes of a length, in order; npass = 0 when it is not provided.
constexpr int kGenMaxPass = 12;
struct GenPlan {
  int n = 0, npass = 0;
  int radix[kGenMaxPass] = {};
  // per pass: points transformed so far, butterflies, twiddle step, 1/ns
  int ns[kGenMaxPass] = {}, nb[kGenMaxPass] = {}, step[kGenMaxPass] = {};
  float inv[kGenMaxPass] = {};
};
GenPlan general_plan(int n);

struct GenArgs {
  const float2* in;   // wave read (may alias out)
  float2* out;        // wave written
  const float* V;     // rows: potential slice (multiplying passes)
  float sigma;
  int nx, ny;
  // the band: columns [0, cpos) and [nx - cneg, nx), rows of the column
  // spectrum [0, rpos) and [ny - rneg, ny)
  int cpos, cneg, rpos, rneg;
  const float2* tw;            // roots of this pass's length (unit_roots)
  const float2 *px, *py;       // propagator factors (unit modulus)
  const float *kx, *ky;
  float k2_lt;                 // band limit on k^2 (see band_limit_thresholds)
  float scale, scale_lo;       // 1/N as the sum of two floats
  GenPlan plan;
};

enum GenRowFlags : int { G_INV = 1, G_MULT = 2, G_FWD = 4 };
// flags: G_INV (band in, real space out), G_MULT | G_FWD (real space in, band
// out) or all three.
cudaError_t launch_general_rows(const GenArgs& a, int flags, cudaStream_t s);
cudaError_t launch_general_columns(const GenArgs& a, cudaStream_t s);

}  // namespace ms
