"""The integer log-sum-exps of the FP64 kernels (csrc/acg_fx.cuh), compiled on
the host and checked against extended precision: the exponential over the range
of its integer form, and sums (whole, and merged from parts) over scales that
stay in that form, cross its limit of 2^14, or lie beyond it."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "application_classification_gb300" / "csrc"

PROBE = r"""
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <limits>
#include <random>
#include <vector>
#include "acg_fx.cuh"
using namespace acg;
static const long double kLn2 = 0.693147180559945309417232121458176568L;
static long double pair_log(const FxLse& a) {
  double m, s;
  fx_pair(a, m, s);
  return (long double)m + logl((long double)s);
}
int main(int argc, char** argv) {
  std::mt19937_64 g(5);
  if (argc == 2) {  // exp over [-R, R]: the largest relative error
    const double R = std::atof(argv[1]);
    std::uniform_real_distribution<double> u(-R, R);
    double worst = 0;
    for (int i = 0; i < 60000; ++i) {
      const double x = i == 0 ? 0.0 : i == 1 ? -0.0 : i == 2 ? 5e-324 : i == 3 ? R : i == 4 ? -R : u(g);
      int k;
      const uint64_t f = fx_exp(fx_bits(x), k);
      const long double e = expl((long double)x - (long double)k * kLn2);
      worst = std::fmax(worst, (double)fabsl(ldexpl((long double)f, -61) / e - 1));
      if (std::fabs(x) < 1000) {  // as a double: half a last place more
        const long double w = expl((long double)x), r = (long double)fx_expd(x);
        if (w > 0x1p-1000L && w < 0x1p1023L && fabsl(r / w - 1) > 4e-16L + (long double)std::fabs(x) * 0x1p-63L) worst = 1;
      }
    }
    // the table form of fixed-point values, every scale in use
    static uint64_t tab[kFxTable];
    for (int j = 0; j < kFxTable; ++j) tab[j] = fx_table_entry(j);
    double worst_tab = 0;
    for (int Q = 47; Q <= 50; ++Q)
      for (int i = 0; i < 20000; ++i) {
        const double x = i == 0 ? 0.0 : i == 1 ? R : i == 2 ? -R : u(g);
        if (std::fabs(x) >= std::ldexp(1.0, 60 - Q)) continue;
        int k;
        const int64_t X = fx_from_double(x, Q);
        const uint64_t f = fx_exp_scaled(X, Q, fx_scaled_factor(Q), tab, k);
        const long double e = expl((long double)X * ldexpl(1.0L, -Q) - (long double)k * kLn2);
        worst_tab = std::fmax(worst_tab, (double)fabsl(ldexpl((long double)f, -61) / e - 1));
        // back to a double: exact where 53 bits hold it, and |X / 2^Q - x| < 2^-Q
        if (std::fabs(fx_to_double(X, Q) - x) > std::ldexp(1.0, -Q) + std::fabs(x) * 0x1p-53) worst_tab = 1;
      }
    std::printf("%.3e %.3e\n", worst, worst_tab);
    return 0;
  }
  // sums of n values N(mean, sd): "error value wide" whole, then merged from parts
  const int n = std::atoi(argv[1]), parts = std::atoi(argv[4]);
  const double mean = std::atof(argv[2]), sd = std::atof(argv[3]);
  std::normal_distribution<double> d(mean, sd);
  std::vector<double> v(n);
  for (double& x : v) x = d(g);
  double m = -std::numeric_limits<double>::infinity();
  for (double x : v) m = std::fmax(m, x);
  long double s = 0;
  for (double x : v) s += expl((long double)x - (long double)m);
  const long double want = (long double)m + logl(s);
  FxLse a, t;
  fx_init(a);
  fx_init(t);
  static uint64_t tab[kFxTable];
  for (int j = 0; j < kFxTable; ++j) tab[j] = fx_table_entry(j);
  for (int i = 0; i < n; ++i)
    if (i % 2) fx_add(a, v[i], tab);
    else fx_add(a, v[i]);
  fx_add(a, -std::numeric_limits<double>::infinity());  // neither adds anything
  fx_add(a, std::numeric_limits<double>::quiet_NaN());
  for (int p = 0; p < parts; ++p) {
    FxLse b;
    fx_init(b);
    for (int i = p; i < n; i += parts) fx_add(b, v[i]);
    fx_merge(t, b);
  }
  FxLse empty;
  fx_init(empty);
  fx_merge(t, empty);
  double em, es;
  fx_pair(empty, em, es);
  std::printf("%.3e %.3e %.17g %d %d\n", (double)fabsl(pair_log(a) - want),
              (double)fabsl(pair_log(t) - want), (double)want, (int)fx_wide(a),
              (int)(em == -std::numeric_limits<double>::infinity() && es == 0.0));
  return 0;
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("fx")
    (d / "probe.cpp").write_text(PROBE)
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", str(CSRC), str(d / "probe.cpp"), "-o", str(d / "probe")],
                   check=True, capture_output=True)
    return d / "probe"


def _out(probe, *args):
    return subprocess.run([str(probe), *map(str, args)], check=True, capture_output=True, text=True).stdout.split()


# The series is cut after r^6 (|r| < 0.0055 + what x's 23-bit float leaves:
# below 1e-16 together), its 32-bit tail loses at most 2^-39 r^2 per step, and
# the 60-bit reduction 2^-59: 2.5e-16 in all.  Beyond |x| = 1000 the reference's
# own k ln 2 in 64 bits adds |x| 2^-64.
@pytest.mark.parametrize("r", [1e-300, 1e-9, 0.004, 0.5, 40.0, 709.0, 16383.999])
def test_exp(probe, r):
    worst, table = map(float, _out(probe, r))
    assert worst <= 2.5e-16 + r * 2.0**-63
    assert table <= 2.5e-16 + r * 2.0**-63  # (|r| < 4e-4 there: cut after r^4, 2^-56)


# An exponential's 2.5e-16, one truncation of 2^-61 of the largest term per
# value, and the (m, s) pair's rounding (2^-52) or, in the wide form, FP64
# rounding of each addition.
@pytest.mark.parametrize("n,mean,sd,parts", [
    (1, -3.0, 1.0, 1), (2, 0.0, 1e-3, 2), (33, -20.0, 40.0, 32), (20000, -120.0, 30.0, 7),
    (5000, 0.0, 0.0, 3), (3000, -16000.0, 300.0, 4), (3000, 16384.0, 1.0, 4), (100, -1e9, 1e8, 5),
    (50, 1e300, 1e299, 3),
])
def test_sum(probe, n, mean, sd, parts):
    whole, merged, want, wide, empty = _out(probe, n, mean, sd, parts)
    bound = 2.5e-16 + n * 2.0**-61 + 2.0**-51 + 2.0**-53 * abs(float(want))
    if int(wide):
        bound += n * 2.0**-52
    assert float(whole) <= bound and float(merged) <= bound + (n * 2.0**-52 if int(wide) else 0)
    assert int(empty) == 1
