// fz_wave.h -- the update constants of the characteristic form in the field precision.
#pragma once
#include <cmath>
#include <limits>

namespace fz {

// p changes by dt_p per difference of the characteristics p +- z0 q, a velocity q by dt_v per sum:
// exactly dt c / 2h, rho c and dt / 2 rho h. A wave's speed follows their product, (dt c / 2h)^2, so the
// rounding of the three constants is a phase error that grows with every step (6.5e-8 of the speed
// squared for the 2D legacy scheme's default grid: 1e-6 of the field after 400 steps). Each constant is
// therefore taken as the nearest value or one of its neighbours, whichever combination leaves the
// smallest error in the product (typically a few 1e-9) and, with less weight, in the impedance.
inline void wave_constants(double dt, double c, double h, double rho, double* z0, double* dt_p, double* dt_v) {
  *z0 = rho * c;
  *dt_p = 0.5 * dt * c / h;
  *dt_v = 0.5 * dt / (h * rho);
}
inline void wave_constants(double dt, double c, double h, double rho, float* z0, float* dt_p, float* dt_v) {
  double z, p, v;
  wave_constants(dt, c, h, rho, &z, &p, &v);
  const auto near = [](double x, int step) {
    const float f = (float)x;
    return step == 0 ? f : std::nextafterf(f, step > 0 ? std::numeric_limits<float>::max() : 0.0f);
  };
  double best = std::numeric_limits<double>::max();
  for (int a = -1; a <= 1; a++)
    for (int b = -1; b <= 1; b++)
      for (int d = -1; d <= 1; d++) {
        const float fz = near(z, a), fp = near(p, b), fv = near(v, d);
        const double ez = (double)fz / z, ep = (double)fp / p, ev = (double)fv / v;
        const double cost = std::fabs(ez * ep * ev - 1.0) + 0.1 * std::fabs(ez * ep / ev - 1.0);
        if (cost < best) {
          best = cost;
          *z0 = fz;
          *dt_p = fp;
          *dt_v = fv;
        }
      }
}

}  // namespace fz
