"""The fixed-point distances of the FP64 cost matrices (csrc/acg_fx.cuh), compiled on
the host, against extended precision: over feature counts and distributions
(N(0, 1), one feature many times the others, lognormal, tight data beside an
outlier) their error, in units of the last place, is no larger than that of the
FP64 form (differences, fused squares, root), on the pairs just above the limit
below which FP64 takes over as on all of them."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "application_classification_gb300" / "csrc"

PROBE = r"""
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "acg_fx.cuh"
using namespace acg;
struct Err {
  double sum2 = 0, max = 0;
  long n = 0;
  void add(double e) { sum2 += e * e; max = std::fmax(max, std::fabs(e)); ++n; }
  double rms() const { return n ? std::sqrt(sum2 / n) : 0; }
};
template <int KM>
void run(int K, const char* dist, double scale) {
  std::mt19937_64 g(K);
  std::normal_distribution<double> n(0, 1);
  const int P = 32, R = 8000;
  auto draw = [&](int i, int k) {
    double x = n(g);
    if (dist[0] == 'l') x = std::exp(scale * x);
    if (dist[0] == 'c' && k == 0) x *= scale;
    if (dist[0] == 'o' && i == 0) x *= scale;  // (in the first row)
    return x;
  };
  std::vector<double> x((size_t)R * K), y((size_t)P * K);
  for (int q = 0; q < P; ++q) for (int k = 0; k < K; ++k) y[(size_t)q * K + k] = draw(-1, k);
  for (int r = 0; r < R; ++r) for (int k = 0; k < K; ++k) x[(size_t)r * K + k] = draw(r, k);
  double top = 0;
  for (double v : y) top = std::fmax(top, std::fabs(v));
  for (int i = 0; i < 128 * K; ++i) top = std::fmax(top, std::fabs(x[i]));
  const int a = std::ilogb(top) + 2;
  const double unit = std::ldexp(1.0, a - FxWindow<KM>::W);
  Err fx, fp, fxn, fpn;
  long left = 0;
  for (int r = 0; r < R; ++r)
    for (int q = 0; q < P; ++q) {
      uint64_t sh = 0, sl = 0;
      int64_t sc = 0;
      bool big = false;
      double s = 0;
      long double e = 0;
      for (int k = 0; k < K; ++k) {
        const double xv = x[(size_t)r * K + k], yv = y[(size_t)q * K + k], t = xv - yv;
        s = std::fma(t, t, s);
        e += ((long double)xv - yv) * ((long double)xv - yv);
        const FxPart px = fx_part<KM>(xv, a, &big), py = fx_part<KM>(yv, a, &big);
        const int32_t h = px.h - py.h, l = px.l - py.l;
        sh += (uint64_t)((int64_t)h * h);
        sc += (int64_t)h * l;
        sl += (uint64_t)((int64_t)l * l);
      }
      if (big || fx_small<KM>(sh)) {
        ++left;
        continue;
      }
      const long double want = sqrtl(e);
      const double ulp = std::ldexp(1.0, std::ilogb((double)want) - 52);
      const double e1 = (double)((fx_root<KM>(sh, sc, sl, a) - want) / ulp);
      const double e2 = (double)((std::sqrt(s) - want) / ulp);
      fx.add(e1);
      fp.add(e2);
      if (want < std::ldexp(1.0, FxWindow<KM>::T + 1) * unit) {
        fxn.add(e1);
        fpn.add(e2);
      }
    }
  std::printf("%.4f %.4f %.4f %.4f %ld %.4f %.4f %ld %ld\n", fx.rms(), fp.rms(), fx.max, fp.max, fxn.n,
              fxn.rms(), fpn.rms(), left, (long)P * R);
}
// values at the ends of the window: the sums must not overflow, whatever the signs
template <int KM>
void ends() {
  std::mt19937_64 g(7);
  double worst = 0;
  const double in = std::nextafter(1.0, 0.0);
  for (int t = 0; t < 20000; ++t) {
    uint64_t sh = 0, sl = 0;
    int64_t sc = 0;
    bool big = false;
    long double e = 0;
    for (int k = 0; k < KM; ++k) {
      const uint64_t b = g();
      // +-(1 - 2^-53), or near it, or halves of the lower part's last bits
      double v[2];
      for (int j = 0; j < 2; ++j) {
        v[j] = (b >> (8 * j)) & 2 ? in : in - std::ldexp((double)((b >> (16 + 8 * j)) & 255), -20);
        if (t % 3 == 0 ? j == 1 : (b >> (8 * j)) & 1) v[j] = -v[j];
      }
      const FxPart px = fx_part<KM>(v[0], 0, &big), py = fx_part<KM>(v[1], 0, &big);
      const int32_t h = px.h - py.h, l = px.l - py.l;
      sh += (uint64_t)((int64_t)h * h);
      sc += (int64_t)h * l;
      sl += (uint64_t)((int64_t)l * l);
      e += ((long double)v[0] - v[1]) * ((long double)v[0] - v[1]);
    }
    if (big) worst = 1;  // (53 bits fit the window)
    if (!big && !fx_small<KM>(sh)) worst = std::fmax(worst, (double)fabsl(fx_root<KM>(sh, sc, sl, 0) / sqrtl(e) - 1));
  }
  bool over = false, nan = false, one = false;
  fx_part<KM>(1.0, 0, &over);
  fx_part<KM>(std::nan(""), 0, &nan);
  fx_part<KM>(std::ldexp(in, -3), -3, &one);
  std::printf("%.3e %d %d %d\n", worst, (int)over, (int)nan, (int)one);
}
int main(int argc, char** argv) {
  const int K = std::atoi(argv[1]);
  const int km = (K + 1) / 2 * 2;
#define CASE(KM_) if (km == KM_) { if (argc == 2) ends<KM_>(); else run<KM_>(K, argv[2], std::atof(argv[3])); }
  CASE(2) CASE(4) CASE(6) CASE(8) CASE(10) CASE(14) CASE(16) CASE(18) CASE(32)
  return 0;
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("fxd")
    (d / "probe.cpp").write_text(PROBE)
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(CSRC), str(d / "probe.cpp"), "-o",
                    str(d / "probe")], check=True, capture_output=True)
    return d / "probe"


def _out(probe, *args):
    out = subprocess.run([str(probe), *map(str, args)], check=True, capture_output=True, text=True).stdout.split()
    return [float(x) for x in out]


@pytest.mark.parametrize("dist,scale", [("n", 1.0), ("l", 1.0), ("l", 2.0), ("c", 100.0), ("o", 12.0)])
@pytest.mark.parametrize("k", [2, 3, 4, 5, 8, 10, 13, 16, 17, 32])
def test_error_below_fp64(probe, k, dist, scale):
    rms, rms64, top, top64, near, nrms, nrms64, left, pairs = _out(probe, k, dist, scale)
    assert rms <= rms64 and top <= top64
    if near >= 500:  # (fewer: the two rms are too rough to compare)
        assert nrms <= nrms64
    if dist == "n":  # few pairs are left to FP64
        assert left <= pairs / 256


# sums of exact parts: the root's own rounding (half a last place, 2^-53) and its 58 bits
@pytest.mark.parametrize("k", [2, 4, 6, 8, 10, 16, 18, 32])
def test_ends_of_the_window(probe, k):
    worst, over, nan, one = _out(probe, k)
    assert worst <= 2.0**-53 + 2.0**-57
    assert (over, nan, one) == (1, 1, 0)
