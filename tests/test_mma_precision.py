"""The MMA loop's per-variable arithmetic (csrc/lp_mma_var.cuh), compiled for the host and compared with a
division for each quotient: no further from extended precision (CPU)."""
import os
import subprocess

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <stdio.h>
#include <stdlib.h>
#include "lp_mma_var.cuh"

static double uniform() { return (rand() + 0.5) / (RAND_MAX + 1.0); }
static double logu(double lo, double hi) { return exp(log(lo) + uniform() * (log(hi) - log(lo))); }

template <typename T> struct Plain {   // each quotient a division
  T x, s, e, up, lo, al, be, ux, xl, xa, bx;
  explicit Plain(const MmaVar& v) : x(v.x), s(v.s), e(v.e), up(v.up), lo(v.lo), al(v.al), be(v.be) {
    // the distances are given: what is compared is what follows from them
    ux = v.ux; xl = v.xl; xa = v.xa; bx = v.bx;
  }
  T q(int k, T a) const {
    const T b[8] = {ux, xl, xa, bx, ux * ux, xl * xl, ux * (ux * ux), xl * (xl * xl)};
    return a / b[k];
  }
  T diag(T p, T q_) const { return T(2) * (q(6, p) + q(7, q_)) + q(2, s) + q(3, e); }
};

int main() {
  srand(1);
  const int n = 200000, K = 9;
  double here[K] = {}, plain[K] = {};
  for (int i = 0; i < n; ++i) {
    MmaVar v;
    v.x = uniform();
    v.al = v.x - logu(1e-7, 0.2);
    v.be = v.x + logu(1e-7, 0.2);
    v.lo = v.al - logu(1e-3, 0.5);
    v.up = v.be + logu(1e-3, 0.5);
    v.s = logu(1e-6, 1e6);
    v.e = logu(1e-6, 1e6);
    const double p = logu(1e-6, 1e3), q = logu(1e-6, 1e3);
    v.distances();
    const Plain<double> d(v);
    const Plain<long double> t(v);
    double delx, diagx;
    v.newton(p, q, 1e-3, delx, diagx);
    const double mine[K] = {v.over_ux(p), v.over_xl(p), v.over_xa(p), v.over_bx(p), v.over_ux2(p), v.over_xl2(p),
                            v.over_ux3(p), v.over_xl3(p), diagx};
    for (int k = 0; k < K; ++k) {
      const long double want = k < 8 ? t.q(k, p) : t.diag(p, q);
      const double other = k < 8 ? d.q(k, p) : d.diag(p, q);
      here[k] += (double)((mine[k] - want) * (mine[k] - want) / (want * want));
      plain[k] += (double)((other - want) * (other - want) / (want * want));
    }
  }
  for (int k = 0; k < K; ++k) printf("%.17g %.17g\n", sqrt(here[k] / n), sqrt(plain[k] / n));
}
"""


def test_quotients_are_as_exact_as_divisions(tmp_path):
    """Root mean square errors over 200000 variables: those of divisions, but for the sampling of their
    difference (1 in 1000)."""
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-x", "c++", "-O1", "-std=c++17", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "loadpath_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = np.array([[float(v) for v in line.split()] for line in
                    subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.splitlines()])
    assert out.shape == (9, 2) and (out[:, 1] > 1e-17).all()
    assert (out[:, 0] <= 1.001 * out[:, 1]).all(), out
