"""The short forms of exp and x^y (vhlle_b200/csrc/vh_crmath.cuh) against the
long forms that decide the arguments they give up on: the same bits over
random arguments, arguments near 1, short mantissas (exact and halfway
results), and the ends of the range; and log_short's error bound."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include "vh_crmath.cuh"
using namespace vh::crm;
int main() {
  unsigned long long s = 88172645463325252ull;
  auto next = [&]() { s ^= s >> 12; s ^= s << 25; s ^= s >> 27; return s * 2685821657736338717ull; };
  auto unit = [&]() { return (double)(next() >> 11) * 0x1p-53; };
  auto same = [](double a, double b) { return std::memcmp(&a, &b, sizeof a) == 0 || (a != a && b != b); };
  long bad = 0, gave_up = 0, n = 300000;
  for (long i = 0; i < n; i++) {
    double x = (2 * unit() - 1) * (i % 4 == 0 ? 750. : i % 4 == 1 ? 5. : i % 4 == 2 ? 1e-3 : 1e-12);
    double r;
    if (std::fabs(x) <= 700. && !exp_try({x, 0.}, &r)) gave_up++;
    if (!same(exp_cr(x), exp_long(x))) bad++;
  }
  const double edge[] = {0., -0., 700., -700., 709.7, 710., -746., -745.2, INFINITY, -INFINITY, NAN, 5e-324};
  for (double x : edge) bad += !same(exp_cr(x), exp_long(x));
  const double ys[] = {1.16849, 1.15635, 1.16187, 4.54886, -0.128012, 1.18735, -1.18423, 0.75, 4. / 3.,
                       -0.25, 0.25, 0.5, 8., -8., 3., 1., -1., 2., 0., 8.5};
  double worst = 0.;
  for (long i = 0; i < n; i++) {
    double x = i % 4 == 0 ? std::ldexp(1 + unit(), (int)(unit() * 2040) - 1020)
             : i % 4 == 1 ? unit() * 50
             : i % 4 == 2 ? 1 + (unit() - .5) * std::ldexp(1., -(int)(unit() * 52)) : unit();
    if (i % 5 == 0) {  // a few leading bits only
      unsigned long long u;
      std::memcpy(&u, &x, 8);
      u &= ~((1ull << (next() % 52)) - 1);
      std::memcpy(&x, &u, 8);
    }
    if (!(x > 0.)) continue;
    for (double y : {ys[next() % 20], (2 * unit() - 1) * 8.})
      bad += !same(pow_cr(x, y), pow_long(x, y));
    const dd a = log_short(x), b = log_dd(x);
    worst = std::fmax(worst, std::fabs((a.hi - b.hi) + (a.lo - b.lo)));
  }
  for (double x : {0., -0., -1., -2., 1., 5e-324, 0x1p-1022, (double)INFINITY, (double)NAN, 1.7e308})
    for (double y : ys) bad += !same(pow_cr(x, y), pow_long(x, y));
  std::printf("%ld %ld %a\n", bad, gave_up, worst);
}
"""


@pytest.mark.parametrize("flags", [["-O2"], ["-O2", "-mfma"]])
def test_short_forms_equal_long_forms(tmp_path, flags):
    if "-mfma" in flags and " fma " not in open("/proc/cpuinfo").read():
        pytest.skip("no fma instruction")
    src = tmp_path / "t.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "t")
    subprocess.run(["g++", "-std=c++17", "-ffp-contract=off", *flags, "-I",
                    os.path.join(ROOT, "vhlle_b200", "csrc"), str(src), "-o", exe], check=True)
    bad, gave_up, worst = subprocess.run([exe], check=True, capture_output=True, text=True).stdout.split()
    assert int(bad) == 0
    assert int(gave_up) < 300  # the bound leaves about 2^-13 of the arguments
    assert float.fromhex(worst) < 2. ** -73
