"""Patterns with a hub: stars, parallel edges and self-loops up to the 256 edges a plan
takes, whose sum at one vertex is hundreds of terms, in both precisions against the
numpy model of the algorithm.

Tolerances: 1e-10 relative for FP64; for mixed plans after two iterations 1e-4
absolute (test_gpu_parity.py, test_gpu_wide_side.py) or, of a hub's sum of n
messages of up to about 20, each rounded about three times to FP32,
n * 3 * 20 * 2^-24."""
import numpy as np
import pytest

import kernel_algebra
from application_classification_gb300 import matcher
from application_classification_gb300.graph import Graph

pytestmark = pytest.mark.gpu


def _graphs(pn, pe, kind, dn=3001, k=4):
    rng = np.random.default_rng(pn + pe)
    ends = lambda n, m: rng.integers(0, n, size=m).astype(np.uint64)  # noqa: E731
    d = Graph(rng.normal(size=(dn, k)), rng.normal(size=(4 * dn, k)), ends(dn, 4 * dn), ends(dn, 4 * dn))
    i = np.arange(pe)
    if kind == "star":  # out to every other vertex, back from it, again
        s, t = (i % 2) * (1 + i // 2 % (pn - 1)), (1 - i % 2) * (1 + i // 2 % (pn - 1))
    elif kind == "parallel":
        s, t = 0 * i, 1 + 0 * i
    else:
        s, t = 0 * i, 0 * i
    p = Graph(rng.normal(size=(pn, k)), rng.normal(size=(pe, k)), s.astype(np.uint64), t.astype(np.uint64))
    return d, p


@pytest.mark.parametrize("kind", ["star", "parallel", "loops"])
@pytest.mark.parametrize("pn,pe", [(30, 58), (65, 128), (128, 254), (128, 256), (2, 256), (100, 205)])
def test_hub(cuda, pn, pe, kind):
    d, p = _graphs(pn, pe, kind)
    ref = kernel_algebra.match(d, p, 2)
    mu = matcher.match(d, p, "fp64", num_iters=2)
    assert np.abs(mu - ref).max() <= 1e-10 * max(1.0, np.abs(ref).max())
    degree = np.bincount(np.concatenate([p.srcs, p.dsts]).astype(int)).max()
    mixed = matcher.match(d, p, "mixed", num_iters=2)
    assert np.abs(mixed - ref).max() <= max(1e-4, degree * 60 * 2.0**-24)
