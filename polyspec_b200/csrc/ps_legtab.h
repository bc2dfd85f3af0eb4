// Coefficients of the FP64 Legendre recurrences (leg_tables_f64), on host and device.
//
// In lam_l = gam_l mu_l with the unit second coefficient, gam_{l+1} = C_l gam_{l-1}, C_l = A_l / A_{l-1}, and
// gam_{l0} = gam_{l0+1} = 1 at l0 = max(m, s).  So gam_l gam_{l+1} = A_l / A_{l0}, and
//   c_l = A_l gam_l / gam_{l+1} = A_{l0} gam_l^2,  d_l = c_l m s / (l (l + 1)),
// where gam_l^2 is a product of rational numbers,
//   C_l^2 = (2l+3) (l+1)^2 (l^2-m^2) (l^2-s^2) / ((2l-1) l^2 ((l+1)^2-m^2) ((l+1)^2-s^2)),
//   A_{l0}^2 = (2l0+3) (l0+1)^2 / ((l0+1)^2 - min(m,s)^2),
// kept here as the sum of two doubles (Dekker 1971), so that c, d and gam are rounded once.  As a chain of plain FP64
// products and quotients they were 2 to 4 roundings off.  Relative rms error of a whole transform against 80-bit sums at the
// same ring positions, with a_l, b_l of each l by themselves (no tables) / the plain chain / this one: spin 0 synthesis
// Nside 64, lmax 128 2.9 / 3.2 / 2.8e-15; spin 1 synthesis Nside 128, lmax 256 7.1 / 7.5 / 6.1e-15; spin 2 adjoint Nside
// 128, lmax 383 15.2 / 15.7 / 13.6e-15.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define PS_HD __host__ __device__ __forceinline__
#else
#define PS_HD inline
#endif

namespace ps {

struct DD {
  double h, l;  // h + l, |l| at most half an ulp of h
};
#ifdef __CUDA_ARCH__  // roundings as written, not contracted
PS_HD double mul_rn(double a, double b) { return __dmul_rn(a, b); }
PS_HD double add_rn(double a, double b) { return __dadd_rn(a, b); }
#else
PS_HD double mul_rn(double a, double b) { return a * b; }
PS_HD double add_rn(double a, double b) { return a + b; }
#endif
PS_HD DD dd_sum(double a, double b) {  // |a| >= |b|
  const double s = add_rn(a, b);
  return {s, add_rn(b, -add_rn(s, -a))};
}
PS_HD DD dd_prod(double a, double b) {
  const double p = mul_rn(a, b);
  return {p, fma(a, b, -p)};
}
PS_HD DD dd_mul(DD a, DD b) {
  const DD p = dd_prod(a.h, b.h);
  return dd_sum(p.h, add_rn(p.l, fma(a.h, b.l, mul_rn(a.l, b.h))));
}
PS_HD DD dd_div(DD a, DD b) {
  const double q = a.h / b.h;
  const double r = add_rn(fma(-q, b.h, a.h), fma(-q, b.l, a.l));
  return dd_sum(q, r / b.h);
}
PS_HD DD dd_sqrt(DD a) {
  const double s = sqrt(a.h);
  return dd_sum(s, add_rn(fma(-s, s, a.h), a.l) / (2.0 * s));
}

// c, d and gam of one (m, s), l by l from l0 on
struct LegChain {
  double m, s, l;
  DD a0, g, next;  // A_{l0}, gam_l^2, gam_{l+1}^2
  PS_HD LegChain(int m_, int s_) : m(m_), s(s_), l(m_ > s_ ? m_ : s_) {
    const double lo = m_ > s_ ? s : m, p = l + 1.0;
    a0 = dd_sqrt(dd_div(dd_prod(2.0 * l + 3.0, p * p), {(p - lo) * (p + lo), 0.0}));
    g = next = {1.0, 0.0};
  }
  PS_HD void values(double& c, double& d, double& gam) const {
    const DD cc = dd_mul(a0, g);
    c = cc.h;
    d = dd_div(dd_mul(cc, {m * s, 0.0}), {s > 0.0 ? l * (l + 1.0) : 1.0, 0.0}).h;
    gam = dd_sqrt(g).h;
  }
  PS_HD void step() {
    l += 1.0;
    const double p = l + 1.0;
    DD n = {(2.0 * l + 3.0) * ((l - m) * (l + m)), 0.0}, d = {(2.0 * l - 1.0) * ((p - m) * (p + m)), 0.0};
    if (s > 0.0) {
      n = dd_mul(n, dd_prod(p * p, (l - s) * (l + s)));
      d = dd_mul(d, dd_prod(l * l, (p - s) * (p + s)));
    }
    const DD g2 = dd_div(dd_mul(g, n), d);
    g = next;
    next = g2;
  }
};

}  // namespace ps
