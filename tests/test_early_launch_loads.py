"""Kernels that may start before their predecessor has finished (those that call
dep_wait) read what the kernels of a match write by ordinary loads: __ldg and
const __restrict__ pointers, whose loads the compiler may move ahead of the wait,
are for arrays that are complete before a match begins (the graph, the features, the
work lists, the pattern).  A check of the sources."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "application_classification_gb300" / "csrc"

# written when a data graph or a plan is made, or by the caller
FIXED = {
    "a.items", "a.wsplit", "a.src_of", "a.row_of", "a.eid", "a.row", "a.qlim_col", "a.pheavy", "a.hcount",
    "a.hbase", "a.hvert", "a.iters_p", "a.d_off", "a.s_off",
    "xr", "x0", "x", "y",  # feature rows
}
FIXED_PARAMS = {"hbase", "hcount", "hvert"}


def _functions():
    """(file, name, parameters, body) of every function of the device sources."""
    for path in sorted(CSRC.glob("*.cu")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        text = re.sub(r"__launch_bounds__\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)", "", text)
        for m in re.finditer(r"([A-Za-z_]\w*)\s*\(([^;{}]*)\)\s*\{", text):
            depth, i = 1, m.end()
            while depth and i < len(text):
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            yield path.name, m.group(1), m.group(2), text[m.end():i]


def test_loads_of_early_kernels():
    funcs = list(_functions())
    early = {(f, n) for f, n, _, body in funcs if re.search(r"\bdep_wait\(\)", body)
             and n not in ("if", "for", "while", "switch")}
    assert len(early) >= 10, early
    # and the functions of the same file that they call
    called = set(early)
    for _ in range(3):
        for f, n, _, body in funcs:
            if (f, n) in called:
                called |= {(f2, n2) for f2, n2, _, _ in funcs
                           if f2 == f and re.search(rf"\b{n2}\s*(<[^;(]*>)?\s*\(", body)}
    bad = []
    for f, n, params, body in funcs:
        if (f, n) not in called or n in ("if", "for", "while", "switch"):
            continue
        for m in re.finditer(r"__ld(g|cs|cv|lu)\s*\(\s*([^;]*)", body):
            arg = m.group(2)
            base = re.match(r"(?:reinterpret_cast<[^>]*>\()?\s*([A-Za-z_][\w.]*)", arg).group(1)
            if base not in FIXED or "reinterpret_cast" in arg.split(")")[0]:
                bad.append((f, n, arg[:60]))
        if (f, n) in early:
            for m in re.finditer(r"__restrict__\s+(\w+)", params):
                if m.group(1) not in FIXED_PARAMS:
                    bad.append((f, n, m.group(0)))
    assert not bad, bad
