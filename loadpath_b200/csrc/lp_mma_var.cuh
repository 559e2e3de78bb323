// One variable of the MMA subproblem (loadpath/mma.py:114-214): its bounds, asymptotes and point, and what the
// passes of the device loop (lp_mma.cu) form from them. Compiles for the host too.
#pragma once
#include "lp_quotient.cuh"

// Quotients that share a divisor share its inverse, corrected (lp_quotient): with a division each the
// float64 units took longer than the memory. A distance of zero (a variable whose bounds meet) gives NaNs, as
// the infinities of its divisions did in the sums.
struct MmaVar {
  double x, s, e, up, lo, al, be;   // the point x, xsi, eta; asymptotes and bounds
  double ux, xl, xa, bx, iux, ixl, ixa, ibx;
  LP_HD void distances() {
    ux = up - x;
    xl = x - lo;
    xa = x - al;
    bx = be - x;
    iux = 1.0 / ux;
    ixl = 1.0 / xl;
    ixa = 1.0 / xa;
    ibx = 1.0 / bx;
  }
  LP_HD double over_ux(double a) const { return lp_quotient(a, ux, iux); }
  LP_HD double over_xl(double a) const { return lp_quotient(a, xl, ixl); }
  LP_HD double over_xa(double a) const { return lp_quotient(a, xa, ixa); }
  LP_HD double over_bx(double a) const { return lp_quotient(a, bx, ibx); }
  LP_HD double over_ux2(double a) const { return lp_quotient(a, ux * ux, iux * iux); }
  LP_HD double over_xl2(double a) const { return lp_quotient(a, xl * xl, ixl * ixl); }
  LP_HD double over_ux3(double a) const { return lp_quotient(a, ux * (ux * ux), iux * (iux * iux)); }
  LP_HD double over_xl3(double a) const { return lp_quotient(a, xl * (xl * xl), ixl * (ixl * ixl)); }
  // delx and diagx at plam, qlam
  LP_HD void newton(double plam, double qlam, double epsi, double& delx, double& diagx) const {
    delx = over_ux2(plam) - over_xl2(qlam) - over_xa(epsi) + over_bx(epsi);
    diagx = 2.0 * (over_ux3(plam) + over_xl3(qlam)) + over_xa(s) + over_bx(e);
  }
  // the direction (dx, dxsi, deta) from gp, gq = P.dlam, Q.dlam
  LP_HD void direction(double plam, double qlam, double gp, double gq, double epsi, double& dx, double& ds,
                       double& de) const {
    double delx, diagx;
    newton(plam, qlam, epsi, delx, diagx);
    const double gtl = over_ux2(gp) - over_xl2(gq);   // (GG^T dlam)_j
    dx = -(delx + gtl) / diagx;
    ds = -s + over_xa(epsi) - over_xa(s * dx);
    de = -e + over_bx(epsi) + over_bx(e * dx);
  }
};
