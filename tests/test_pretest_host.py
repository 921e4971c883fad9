"""The FP32 pre-test's msq and error bound (phs_pretest.h, compiled as host C++) against the map in
FP64 and in long double, with the hardware sine, cosine, exponential and quotient replaced by
functions that are wrong by their documented bounds: resonances of m Gamma / s from 1e-1 to 1e-10,
exponential maps, and x up to the last double below 1."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gpu_phs_gb300", "csrc")

DRIVER = r"""
#include <cstdio>
#include <cmath>
#include <random>
#include "phs_pretest.h"
typedef long double Q;
static const Q HALF_PI = 1.57079632679489661923132169163975144L;
long n = 0, bad = 0;
double worst = 0;
static void hold(float m, float e, double f64, Q exact) {
  n++;
  for (Q v : {(Q)f64, exact}) {
    if (!(v == v) || !(std::fabs((double)v) < 1e30)) continue;
    const double d = std::fabs((double)(v - (Q)m)) / (double)e;
    worst = std::fmax(worst, d);
    bad += !(d <= 1) && e == e;   // NaN bounds decide nothing
  }
}
int main() {
  std::mt19937_64 g(7);
  std::uniform_real_distribution<double> U(0, 1);
  auto draw = [&](int i) {
    switch (i % 4) {
      case 0: return U(g);
      case 1: return 1.0 - std::ldexp(U(g), -(int)(U(g) * 53));
      case 2: return std::ldexp(U(g), -(int)(U(g) * 53));
      default: return 1.0 - (1 + (int)(U(g) * 64)) * 0x1p-53;
    }
  };
  for (double E : {1000.0, 13000.0})
    for (double m : {1.0, 80.4, 125.0, 500.0})
      for (int lg = 1; lg <= 10; lg++) {
        const double s = E * E, mw = s * std::pow(10.0, -lg), w = mw / m;
        if (w > 0.3 * m) continue;
        for (double mn : {0.0, 0.3 * m * m}) {
          const double mx = s, a0 = std::atan((mn - m * m) / (m * w)), a1 = std::atan((mx - m * m) / (m * w));
          const float c[6] = {(float)a0, (float)(a1 - a0), (float)(HALF_PI + (Q)a0), (float)(HALF_PI - (Q)a1),
                              (float)(m * m), (float)(m * w)};
          for (int i = 0; i < 20000; i++) {
            const double x = draw(i);
            float e;
            const float r = msq_f32(PHS_MAP_SCHANNEL, c[0], c[1], c[2], c[3], c[4], c[5], x, e);
            const double z = (1 - x) * a0 + x * a1;
            const Q ze = (1 - (Q)x) * a0 + (Q)x * a1;
            if (!(std::fabs(z) < (double)HALF_PI)) continue;
            hold(r, e, m * (m + w * std::tan(z)), (Q)m * ((Q)m + (Q)w * tanl(ze)));
          }
        }
      }
  for (double E : {1000.0, 13000.0})
    for (double m : {5.11e-4, 1.0, 10.0})
      for (int t : {PHS_MAP_INFRARED, PHS_MAP_TCHANNEL}) {
        const double mx = E * E, mn = 0, q0 = m * m;
        const double a1 = t == PHS_MAP_TCHANNEL ? 2 * std::log((mx - mn) / (2 * q0) + 1) : std::log((mx - mn) / q0 + 1);
        for (int i = 0; i < 40000; i++) {
          const double x = draw(i);
          float e;
          const float r = msq_f32(t, (float)q0, (float)a1, (float)mn, (float)mx, 0, 0, x, e);
          const bool up = t == PHS_MAP_TCHANNEL && !(x < 0.5);
          const Q y = up ? (1 - (Q)x) * a1 : (Q)x * a1, v = q0 * expl(y) - q0;
          const double y64 = (up ? 1 - x : x) * a1, v64 = q0 * std::exp(y64) - q0;
          hold(r, e, up ? -v64 + mx : v64 + mn, up ? mx - v : v + mn);
        }
      }
  std::printf("%ld %ld %.3f\n", n, bad, worst);
}
"""


@pytest.mark.parametrize("sign", [-1, 0, 1])
@pytest.mark.parametrize("cos_sign", [-1, 1])
def test_interval_holds_the_map(tmp_path, sign, cos_sign):
    try:
        subprocess.run(["g++", "--version"], check=True, capture_output=True)
    except (OSError, subprocess.CalledProcessError):
        pytest.skip("g++ not available")
    head = open(os.path.join(CSRC, "phs_pretest.h")).read()
    for old, new in (("return sinf(a);", f"return sinf(a) + ({sign}) * 3.6e-7f;"),
                     ("return cosf(a);", f"return cosf(a) + ({cos_sign}) * 4.1e-7f;"),
                     ("return expf(a);", f"return expf(a) * (1.0f + ({sign}) * (2.0f + 1.2f * fabsf(a)) * 6e-8f);"),
                     ("return a / b;", f"return a / b * (1.0f + ({sign}) * 2.4e-7f);")):
        assert head.count(old) == 1
        head = head.replace(old, new)
    (tmp_path / "phs_pretest.h").write_text(head)
    (tmp_path / "t.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-std=gnu++17", "-I", str(tmp_path), "-I", CSRC,
                    str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    n, bad, worst = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout.split()
    assert int(n) > 500_000
    assert int(bad) == 0, worst
