"""FP64 matches on graphs where many vertices lie far from every pattern edge (a
single out-edge whose distances are far beyond the fixed-point stage's range, or
beyond the integer log-sum-exps' too), beside ordinary vertices in the same
stages, against the FP64 numpy model of the algorithm.

Tolerance: the FP64 path's, 1e-10 relative to max|mu| (test_gpu_parity.py)."""
import numpy as np
import pytest

import kernel_algebra
from application_classification_gb300 import matcher
from application_classification_gb300.graph import Graph

pytestmark = pytest.mark.gpu

REL = 1e-10


def _graphs(dn, pn, pe, far, every, first, seed=1, k=8):
    """A pattern planted among the vertices other than first, first + every, ...;
    those have one out-edge, `far` to 5 `far` from every pattern edge."""
    rng = np.random.default_rng(seed)
    lone = np.arange(first, dn, every)
    plain = np.setdiff1d(np.arange(dn), lone)
    at = rng.choice(plain, size=pn, replace=False)
    ps, pd = rng.integers(0, pn, size=pe), rng.integers(0, pn, size=pe)
    srcs = np.concatenate([lone, at[ps], rng.choice(plain, size=3 * dn)])
    dsts = np.concatenate([rng.integers(0, dn, size=lone.size), at[pd], rng.integers(0, dn, size=3 * dn)])
    nf, ef = 2 * rng.normal(size=(dn, k)), 2 * rng.normal(size=(srcs.size, k))
    pef = ef[lone.size:lone.size + pe] + 0.05 * rng.normal(size=(pe, k))
    ef[: lone.size] *= (far * rng.uniform(1.0, 5.0, lone.size) / np.linalg.norm(ef[: lone.size], axis=1))[:, None]
    order = rng.permutation(srcs.size)
    u64 = lambda x: np.ascontiguousarray(x, dtype=np.uint64)  # noqa: E731
    d = Graph(nf, ef[order], u64(srcs[order]), u64(dsts[order]))
    p = Graph(nf[at] + 0.05 * rng.normal(size=(pn, k)), pef, u64(ps), u64(pd))
    return d, p


# groups of one, two and four warps; enough vertices for many stages a group;
# far vertices first, second or alternately in their stage of two
@pytest.mark.parametrize("far", [1.1e3, 2e4, 1e8])
@pytest.mark.parametrize("every,first", [(3, 0), (2, 0), (2, 1)])
@pytest.mark.parametrize("dn,pn,pe", [(60000, 16, 30), (30000, 40, 50), (12000, 40, 100), (6000, 70, 200)])
def test_far_vertices(cuda, dn, pn, pe, every, first, far):
    d, p = _graphs(dn, pn, pe, far, every, first)
    ref = kernel_algebra.match(d, p, 3)
    mu = matcher.match(d, p, "fp64", num_iters=3)
    assert np.isfinite(mu).all()
    assert np.abs(mu - ref).max() <= REL * max(1.0, np.abs(ref).max())
