"""Shared memory of the vertex phases that share a stage between warps
(csrc/acg_vschedule.h), on the host: for every pattern that a plan takes (up to 128
vertices and 256 edges, hubs, parallel edges and self-loops included) the kernel the
launch chooses fits a block's 227 KB; only where four warps share an FP64 stage does
the schedule have to stay in global memory, and wide FP32 patterns whose schedule does
not fit are beyond the terms a lane that the kernel is given (kWideTerms)."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "application_classification_gb300" / "csrc"

PROBE = r"""
#include <cstdio>
#include <random>
#include <vector>
#include "acg_vschedule.h"
using namespace acg;
static int pad(int x, int m) { return (x + m - 1) / m * m; }
// build_incidence's layout
static std::vector<int> incidence(int pn, const std::vector<int>& s, const std::vector<int>& d) {
  const int pe = (int)s.size();
  std::vector<int> v(s);
  v.insert(v.end(), d.begin(), d.end());
  for (const std::vector<int>* e : {&d, &s}) {
    std::vector<int> off(pn + 1, 0), q;
    for (int x : *e) ++off[x + 1];
    for (int p = 0; p < pn; ++p) off[p + 1] += off[p];
    for (int p = 0; p < pn; ++p)
      for (int i = 0; i < pe; ++i)
        if ((*e)[i] == p) q.push_back(i);
    v.insert(v.end(), off.begin(), off.end());
    v.insert(v.end(), q.begin(), q.end());
  }
  return v;
}
int main() {
  std::mt19937 g(3);
  long over = 0, global = 0, few = 0, n = 0, none = 0;
  for (int pn : {1, 2, 31, 33, 64, 65, 100, 125, 127, 128})
    for (int pe : {1, 2, 31, 33, 63, 64, 65, 66, 68, 72, 100, 126, 128, 129, 130, 150, 171, 172, 200, 204, 205, 255, 256})
      for (int kind = 0; kind < 4; ++kind) {
        std::vector<int> s(pe), d(pe);
        for (int i = 0; i < pe; ++i) {
          s[i] = kind == 0 ? g() % pn : kind == 1 ? 0 : kind == 2 ? i % 2 * (i / 2 % pn) : 0;
          d[i] = kind == 0 ? g() % pn : kind == 1 ? 0 : kind == 2 ? (1 - i % 2) * (i / 2 % pn) : i % pn;
        }
        const std::vector<int> pat = incidence(pn, s, d);
        std::vector<uint32_t> out;
        {
          const int pp = pad(pe, 2), pnp = pad(pn, 2);
          const int nw = pp <= 64 && pn <= 64 ? 1 : pp <= 128 ? 2 : 4;
          const int nt = vertex_warp_schedule(pat.data(), pn, pe, pp, pnp, kFxVps, &out, 32 * nw, 2, 8);
          none += nt == 0;
          size_t b = FxSmem(pn, pe, pp, pnp, nt, nw, false).total;
          if (b > kBlockSmem) {
            ++global;
            few += nw < 4;
            b = FxSmem(pn, pe, pp, pnp, nt, nw, true).total;
          }
          over += b > kBlockSmem;
          ++n;
        }
        const int pp = pad(pe, 4), pnp = pad(pn, 4);
        if (pp > 64) {
          const int nw = pp <= 128 ? 1 : 2, V = 256 / (pp / 4);
          const int nt = vertex_warp_schedule(pat.data(), pn, pe, pp, pnp, kWv, &out, 32 * nw, 4);
          none += nt == 0;
          if (nw == 1 || nt <= KWIDETERMS) over += WideSmem(V, pn, pe, pp, pnp, nt, nw).total > kBlockSmem;
          ++n;
        }
      }
  std::printf("%ld %ld %ld %ld %ld\n", over, few, none, global, n);
  return 0;
}
"""


def test_every_pattern_fits(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("needs g++")
    terms = re.search(r"constexpr int kWideTerms = (\d+);", (CSRC / "acg_vertex_wide.cu").read_text()).group(1)
    (tmp_path / "probe.cpp").write_text(PROBE.replace("KWIDETERMS", terms))
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", str(CSRC), str(tmp_path / "probe.cpp"), "-o",
                    str(tmp_path / "probe")], check=True, capture_output=True)
    out = subprocess.run([str(tmp_path / "probe")], check=True, capture_output=True, text=True).stdout
    over, few, none, in_global, n = map(int, out.split())
    assert (over, few, none) == (0, 0, 0)
    assert 0 < in_global < n // 10
