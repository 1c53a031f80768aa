"""FP64 cost matrices: equal rows have equal costs wherever they stand in the graph
(maxima and their first-of-equals rule rest on exact ties), among ordinary rows and
among rows of another scale."""
import numpy as np
import pytest

from application_classification_gb300 import matcher
from application_classification_gb300.graph import Graph

pytestmark = pytest.mark.gpu


# With zero iterations mu is the vertex cost matrix, negated and normalised by
# column constants: equal costs, equal bits.
@pytest.mark.parametrize("kv", [2, 5, 13, 32])
@pytest.mark.parametrize("scale", [1.0, 9.0, 300.0])
def test_equal_rows(cuda, kv, scale):
    rng = np.random.default_rng(kv)
    n, kinds = 120000, 997
    base = rng.normal(size=(kinds, kv))
    kind = rng.integers(0, kinds, size=n)
    nf = base[kind]
    other = np.zeros(n, dtype=bool)  # rows of another scale: half of every fifth run of 256
    other[np.arange(n) % 1280 < 128] = True
    nf[other] *= scale
    ends = lambda m, k: rng.integers(0, m, size=k).astype(np.uint64)  # noqa: E731
    d = Graph(nf, rng.normal(size=(n, 2)), ends(n, n), ends(n, n))
    p = Graph(0.5 * rng.normal(size=(9, kv)), rng.normal(size=(12, 2)), ends(9, 12), ends(9, 12))
    mu = matcher.match(d, p, "fp64", num_iters=0)
    assert np.isfinite(mu).all()
    for rows in (~other, other):
        first = np.full(kinds, -1)
        idx = np.flatnonzero(rows)
        first[kind[idx][::-1]] = idx[::-1]
        assert np.array_equal(mu[idx], mu[first[kind[idx]]])
