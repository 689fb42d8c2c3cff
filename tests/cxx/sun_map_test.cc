// The mu_s mapping along a ray (SunCoordinate of atmo_device.cuh) against
// FP64, for planets with the sun down to any zenith angle.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "../../precomputed_atmospheric_scattering_gb300/csrc/atmo_device.cuh"

using namespace atmo;

int main() {
  const double radii[][2] = {{6360.0, 6420.0}, {6360e3, 6420e3}, {3000.5, 3120.25}, {1.0, 1.01}};
  int bad = 0;
  double worst = 0.0;
  for (const auto& r : radii) {
    for (double zenith : {10.0, 30.0, 60.0, 89.0, 102.0, 120.0, 180.0}) {
      const double Rb = r[0], Rt = r[1], H = std::sqrt(Rt * Rt - Rb * Rb), d_min = Rt - Rb;
      const double mu_min = std::cos(zenith * kPiD / 180.0);
      const double D = -Rb * mu_min + std::sqrt(Rb * Rb * mu_min * mu_min + H * H);
      const double A = (D - d_min) / (H - d_min), t = d_min / (H - d_min);
      Consts c;
      Shape s;
      std::memset(&c, 0, sizeof c);
      std::memset(&s, 0, sizeof s);
      c.Rb = (float)Rb;
      c.Rt = (float)Rt;
      c.H = (float)H;
      c.mus_A = (float)A;
      s.smus = 32;
      const SunMap m = MakeSunMap(c, s);
      for (int i = 0; i <= 20000; ++i) {
        const float rmus = (float)(Rb * (mu_min + (1.0 - mu_min) * i / 20000.0));
        const double y = std::sqrt((double)rmus * rmus + H * H) + std::fabs((double)rmus);
        const double a = std::max(((rmus > 0.0f ? H * H / y : y) - d_min) / (H - d_min), 0.0);
        const double x = std::max(1.0 - a / A, 0.0) / (1.0 + a);
        // In units of 2^-24: the distance to the top, whose factors round five
        // times (three of them H^2's), moves a by 5 (a + t); the quotients by
        // the range and A by 3 a; numerator, denominator, reciprocal and
        // product round once each.  The radii as floats move t by 2 Rt / d_min
        // of its own, where they are not exact.
        const double radius = (c.Rb == Rb && c.Rt == Rt) ? 0.0 : 4.0 * t * Rt / d_min;
        const double bound = std::ldexp(
            (1.0 + 1.0 / A) * (5.0 * (a + t) + 3.0 * a + radius) / ((1.0 + a) * (1.0 + a)) + 4.0,
            -24);
        const double e = std::fabs(SunCoordinate(m, rmus) - x);
        worst = std::max(worst, e / bound);
        bad += !(e <= bound);
      }
    }
  }
  std::printf("%d wrong, worst %.2f of the bound\n", bad, worst);
  return bad != 0;
}
