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
// kAngle: errors against FP64 after 51 to 52 slices, as a ratio to those of the
// modulus alone, geometric mean over 26 combinations of 17 grids from 64^2 to
// 1024^2 (four with mixed radices), four specimens and both forms of the slice
// loop, and over 13 focal-series losses:
//   kAngle     0.2    0.3    0.4    0.5    0.6    0.7
//   exit wave  0.925  0.865  0.835  0.831  1.084  1.094
//   loss       0.899  0.701  0.694  0.718  1.523  1.501
// 0.4: near both minima and not at the edge.  (Above 0.5 pairs of plain rounding
// come back.)  Single grids scatter: a 512^2 SrTiO3 loss has 0.43e-6 at 0.2 and
// 0.73e-6 at 0.4 (rms of 16 inputs; 0.70e-6 with the modulus alone), a 512^2
// silicon one 1.18e-6 and 0.31e-6.
//
// The angle error is below 1e-6, so its sine, the cross product, is the angle to
// FP64: no inverse function is needed (a 1024^2 grid takes two thousand factors).
inline void unit_fp32(double c, double s, float* co, float* so) {
  constexpr double kAngle = 0.4;
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
