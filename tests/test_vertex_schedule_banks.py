"""The vertex phase's schedule (csrc/acg_vschedule.h) for groups of one, two and
four warps and 4- and 8-byte stage elements: every job's terms stay in the tile
form's order on one lane, no lane holds more terms than longest-first assignment
gives, and a load takes no more shared-memory passes than the jobs in the order of
that assignment do."""
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

from test_vertex_schedule import PROBE

CSRC = Path(__file__).resolve().parents[1] / "application_classification_gb300" / "csrc"


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("needs g++")
    d = tmp_path_factory.mktemp("vbanks")
    src = d / "probe.cpp"
    call = "acg::vertex_warp_schedule(pat.data(), pn, pe, pp, pnp, vps, &w)"
    assert call in PROBE
    src.write_text(PROBE.replace(call, call[:-1] + ", NL, PL, EL)"))

    def make(nl, pl, el):
        exe = d / f"p{nl}_{pl}_{el}"
        subprocess.run([cxx, "-std=c++17", "-O1", f"-DNL={nl}", f"-DPL={pl}", f"-DEL={el}", "-I", str(CSRC),
                        str(src), "-o", str(exe)], check=True, capture_output=True)
        return exe
    return make


def _passes(lanes, elem):
    """Passes of all loads: per step and group of lanes, the busiest bank's words."""
    g = 128 // elem
    total = 0
    for t in range(lanes.shape[1]):
        for l0 in range(0, lanes.shape[0], g):
            offs = np.unique(lanes[l0:l0 + g, t] & 0xFFF)
            total += np.bincount(offs % g).max()
    return total


@pytest.mark.parametrize("pn,pe,vps,nl,pl,elem", [
    (16, 32, 4, 32, 2, 4), (32, 64, 4, 32, 2, 4), (40, 120, 2, 32, 4, 4), (48, 192, 2, 64, 4, 4),
    (33, 64, 4, 32, 2, 8), (40, 100, 2, 64, 2, 8), (64, 250, 1, 128, 2, 8), (1, 2, 4, 32, 2, 4)])
def test_order_balance_and_banks(probe, pn, pe, vps, nl, pl, elem):
    rng = np.random.default_rng(pn * 1000 + pe)
    edges = rng.integers(0, pn, (pe, 2))
    pp, pnp = -(-pe // 4) * 4, -(-pn // 4) * 4
    text = f"1\n{vps} {pn} {pe} {pp} {pnp}\n" + "".join(f"{s} {d}\n" for s, d in edges)
    out = subprocess.run([str(probe(nl, pl, elem))], input=text, check=True, capture_output=True, text=True).stdout.split()
    nt, n = int(out[0]), int(out[1])
    words = np.array(out[2:2 + n], dtype=np.int64)
    assert n == nt * nl and nt % 4 == 0
    lanes = words.reshape(nt // 4, nl, 4).transpose(1, 0, 2).reshape(nl, nt)
    START, END = 1 << 12, 1 << 13
    row = -(-pn // 32) * 32 + 1
    oM, oY, oC = 0, vps * pp, 4 * vps * pp
    job = {}
    for jv in range(vps):
        for p in range(pn):
            job[jv * row + p] = ([oC + jv * pnp + p] + [oM + jv * pp + q for q in range(pe) if edges[q, 1] == p]
                                 + [oY + jv * pp + q for q in range(pe) if edges[q, 0] == p])
    seen = []
    for lane in lanes:
        t = 0
        while t < nt and lane[t] & START:
            slot = int(lane[t]) >> 16
            want = job[slot]
            got = lane[t:t + len(want)]
            assert list(got & 0xFFF) == want and all(got >> 16 == slot)
            assert list((got & START) != 0) == [True] + [False] * (len(want) - 1)
            assert list((got & END) != 0) == [False] * (len(want) - 1) + [True]
            seen.append(slot)
            t += len(want)
        assert not lane[t:].any()
    assert sorted(seen) == sorted(job)
    # longest first (ties: staged vertex, pattern vertex), each to the least loaded lane
    plain = [[] for _ in range(nl)]
    for slot in sorted(job, key=lambda x: (-len(job[x]), x)):
        min(plain, key=len).extend(job[slot])
    longest = max(len(x) for x in plain)
    assert nt == -(-longest // 4) * 4
    ref = np.array([x + [0] * (nt - len(x)) for x in plain])
    assert _passes(lanes, elem) <= _passes(ref, elem)
