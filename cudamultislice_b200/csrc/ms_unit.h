// ms_unit.h -- unit factors in FP32 (host).
#pragma once
#include <cmath>

namespace ms {

// (cos, sin) as the FP32 pair within one ulp of each component with the least
// hypot(|modulus^2 - 1|, angle error / 5).  Unit factors applied once per transform
// or per slice (twiddles, propagator) then scale the wave by |(c, s)|^S over a
// stack of S slices only to that pair's remaining modulus error, far below the
// plain rounding's, which adds up coherently when the slices repeat (crystals).  The
// modulus alone would let the angle be off by more than an ulp: 52 slices of a
// 512^2 crystal then end 0.94e-6 to 1.11e-6 from FP64, with the fifth of the angle
// 0.84e-6 to 0.98e-6, and a focal-series loss 0.94e-6 (rms of 32 inputs) against
// 0.42e-6; a tenth or a half of the angle 0.69e-6 and 1.0e-6.
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
