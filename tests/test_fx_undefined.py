"""The integer arithmetic of csrc/acg_fx.cuh wraps by design, in unsigned types: the
host probes of its other tests run without undefined behaviour (signed overflow,
shifts of negative values or by too much, conversions out of range)."""
import shutil
import subprocess
from pathlib import Path

import pytest

import test_fx_distance
import test_fx_lse
import test_fx_lse_far

CSRC = Path(__file__).resolve().parents[1] / "application_classification_gb300" / "csrc"

RUNS = {
    "lse": (test_fx_lse.PROBE, [["709.0"], ["16383.999"], ["1e-9"], ["2000", "-120.0", "30.0", "7"],
                                ["300", "-16000.0", "300.0", "4"], ["100", "-1e9", "1e8", "5"]]),
    "far": (test_fx_lse_far.PROBE, [["1100.0", "-9.0", "300"], ["1e5", "0.0", "300"], ["1.7e7", "0.0", "300"],
                                    ["1e300", "0.0", "300"]]),
    "distance": (test_fx_distance.PROBE, [["2", "n", "1.0"], ["17", "l", "2.0"], ["32", "c", "100.0"], ["4"],
                                          ["8"], ["16"], ["32"]]),
}


@pytest.mark.parametrize("name", sorted(RUNS))
def test_no_undefined_behaviour(tmp_path, name):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("needs g++")
    probe, runs = RUNS[name]
    (tmp_path / "probe.cpp").write_text(probe)
    flags = ["-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover=undefined"]
    build = subprocess.run([cxx, *flags, "-I", str(CSRC), str(tmp_path / "probe.cpp"), "-o", str(tmp_path / "probe")],
                           capture_output=True, text=True)
    if build.returncode and "ubsan" in build.stderr:
        pytest.skip("needs libubsan")
    assert build.returncode == 0, build.stderr
    for args in runs:
        r = subprocess.run([str(tmp_path / "probe"), *args], capture_output=True, text=True)
        assert r.returncode == 0, (args, r.stderr)
