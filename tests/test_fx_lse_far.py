"""Log-sum-exps (csrc/acg_fx.cuh) whose values lie far apart, compiled on the host
and checked against extended precision: values up to the integer form's limit of
2^24 and beyond it, before, between and after ordinary ones, in the order in
which a stage of the FP64 vertex phase adds them (the fixed-point terms of the
stage first, by fx_add_term; a state found wide at a stage's start takes fx_add).
A state that has met far values has to be back in integer form with the next
ordinary one."""
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
static uint64_t tab[kFxTable];
static long double log_of(const FxLse& a) {
  double m, s;
  fx_pair(a, m, s);
  return (long double)m + logl((long double)s);
}
static long double exact(const std::vector<double>& v) {
  long double m = -INFINITY, s = 0;
  for (double x : v) m = fmaxl(m, x);
  for (double x : v) s += expl((long double)x - m);
  return m + logl(s);
}
int main(int argc, char** argv) {
  for (int j = 0; j < kFxTable; ++j) tab[j] = fx_table_entry(j);
  const double far = std::atof(argv[1]), base = std::atof(argv[2]);
  const int trials = std::atoi(argv[3]), Q = 50;
  const int32_t c = fx_scaled_factor(Q);
  std::mt19937_64 g(11);
  std::normal_distribution<double> n(0, 3);
  std::uniform_real_distribution<double> u(0, 1);
  double worst = 0;
  int still_wide = 0;
  for (int t = 0; t < trials; ++t) {
    FxLse a;  // stages of two values
    fx_init(a);
    std::vector<double> v;
    const int stages = 1 + t % 20;
    for (int i = 0; i < stages; ++i) {
      double x[2];
      bool isfar[2];
      for (int j = 0; j < 2; ++j) {
        isfar[j] = u(g) < 0.3 || (t % 3 == 0 && i == 0);
        // (ordinary values are multiples of 2^-Q: what the fixed-point stage adds)
        x[j] = isfar[j] ? -far * (1 + u(g)) : base + std::ldexp(std::rint(std::ldexp(n(g), Q)), -Q);
        v.push_back(x[j]);
      }
      if (fx_wide(a)) {
        for (int j = 0; j < 2; ++j) fx_add(a, x[j]);
      } else {
        for (int j = 0; j < 2; ++j)
          if (!isfar[j]) {
            int k;
            const uint64_t f = fx_exp_scaled(fx_from_double(x[j], Q), Q, c, tab, k);
            fx_add_term(a, k, f);
          }
        for (int j = 0; j < 2; ++j)
          if (isfar[j]) a = fx_add_far(a, x[j]);
      }
    }
    if (t % 2) {  // an ordinary value last
      v.push_back(base);
      fx_add(a, base, tab);
      still_wide += fx_wide(a);
    }
    const long double w = exact(v);
    const double bound = 2.5e-16 + v.size() * 0x1p-52 + 0x1p-51 + 0x1p-53 * std::fabs((double)w);
    worst = std::fmax(worst, (double)fabsl(log_of(a) - w) / bound);
  }
  std::printf("%.3e %d\n", worst, still_wide);
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


# Errors in units of the bound of test_fx_lse.py: an exponential's 2.5e-16, a
# truncation or an FP64 rounding per value, the pair's and the result's rounding.
@pytest.mark.parametrize("base", [0.0, -9.0])
@pytest.mark.parametrize("far", [30.0, 1100.0, 16000.0, 2.0**14, 1e5, 2.0**23, 2.0**24, 1e9, 1e300])
def test_far(probe, far, base):
    out = subprocess.run([str(probe), repr(far), repr(base), "3000"], check=True, capture_output=True, text=True)
    worst, still_wide = out.stdout.split()
    assert float(worst) <= 1.0
    assert int(still_wide) == 0
