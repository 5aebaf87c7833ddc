// ms_unit.h -- unit factors in FP32 (host).
#pragma once
#include <cmath>

namespace ms {

// (cos, sin) as the FP32 pair within one ulp of each component with the least
// hypot(modulus^2 - 1, kAngle x angle error).  Unit factors applied once per
// transform or per slice (twiddles, propagator) then scale the wave by |(c, s)|^S
// over a stack of S slices only to that pair's remaining modulus error, far below
// the plain rounding's, which adds up coherently when the slices repeat (crystals).
// The modulus alone would let the angle be off by more than an ulp.
//
// kAngle, errors against FP64 after about 50 slices.  As a ratio to those of the
// modulus alone, geometric mean over 26 combinations of 17 grids from 64^2 to
// 1024^2 (four with mixed radices), four specimens and both forms of the slice
// loop, and over 13 focal-series losses:
//   kAngle         0.2    0.3    0.4    0.5    0.6    0.7
//   exit wave      0.925  0.865  0.835  0.831  1.084  1.094
//   loss           0.899  0.701  0.694  0.718  1.523  1.501
// and of single SrTiO3 results, rms of 14 inputs, 1e-6:
//                  0 (modulus)  0.2   0.25  0.3   0.35  0.4
//   512^2  dL/dxy  2.43         1.70  1.60  2.44  2.51  1.82
//          loss    1.10         0.47  0.53  0.30  0.30  0.96
//   256^2  image   0.54         0.50  0.54  0.72  0.64  0.75
// Waves gain a little up to 0.5 (above it pairs of plain rounding come back); what
// is left of a result's bias changes with the table by up to a factor of two either
// way.  0.2 is below the modulus alone in the means and in each of these.
//
// The angle error is below 1e-6, so its sine, the cross product, is the angle to
// FP64: no inverse function is needed (a 1024^2 grid takes two thousand factors).
inline void unit_fp32(double c, double s, float* co, float* so) {
  constexpr double kAngle = 0.2;
  const float cs[3] = {std::nextafter((float)c, -INFINITY), (float)c, std::nextafter((float)c, INFINITY)};
  const float ss[3] = {std::nextafter((float)s, -INFINITY), (float)s, std::nextafter((float)s, INFINITY)};
  double best = INFINITY;
  for (float x : cs)
    for (float y : ss) {
      // the modulus first: its error adds up over all transforms of a run, the
      // angle's partly cancels between a transform and its inverse
      const double n = (double)x * x + (double)y * y - 1.0, a = kAngle * ((double)y * c - (double)x * s);
      const double cost = n * n + a * a;
      if (cost < best) {
        best = cost;
        *co = x;
        *so = y;
      }
    }
}

}  // namespace ms
