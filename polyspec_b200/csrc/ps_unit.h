// Roots of unity for the host's tables.
#pragma once
#include <cmath>
#include <cstdint>

namespace ps {

// c + i s = e^{i pi q / den}, den > 0, to about an ulp.  The angle is reduced to the first octant in whole numbers, and what
// its product with pi and the quotient round off enters to first order: cos(M_PI * q / den) as it stands carries the
// rounding of angles up to 2 pi, 2.0e-16 rms and 1.3e-15 at most over ring lengths up to 4092, this 0.3e-16 and 1.1e-16.
inline void unit_root(int64_t q, int64_t den, double& c, double& s) {
  constexpr double PI_LOW = 1.2246467991473532e-16;  // pi - M_PI
  int64_t r = q % (2 * den);
  if (r < 0) r += 2 * den;
  const bool lower = r > den;
  if (lower) r = 2 * den - r;
  const bool left = 2 * r > den;
  if (left) r = den - r;
  const bool steep = 4 * r > den;
  const double n = double(steep ? den - 2 * r : r), d = double(steep ? 2 * den : den);
  const double p = M_PI * n, plow = std::fma(M_PI, n, -p) + PI_LOW * n;
  const double t = p / d, tlow = (std::fma(-t, d, p) + plow) / d;
  const double ct = std::cos(t), st = std::sin(t);
  const double ca = ct - tlow * st, sa = st + tlow * ct;
  c = steep ? sa : ca;
  s = steep ? ca : sa;
  if (left) c = -c;
  if (lower) s = -s;
}

}  // namespace ps
