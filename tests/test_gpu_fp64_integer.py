"""FP64 plans whose work runs on the integer pipes, against the FP64 numpy model
of the algorithm (kernel_algebra, itself pinned to the reference's golden
outputs): sizes at the edges of the kernels' shapes, and inputs that leave the
integer form's range in whole or in part, where FP64 takes over.

Tolerance: the FP64 path's, 1e-10 relative to max|mu| (test_gpu_parity.py)."""
import numpy as np
import pytest

import kernel_algebra
from application_classification_gb300 import matcher
from application_classification_gb300.graph import Graph

pytestmark = pytest.mark.gpu

REL = 1e-10


def _graphs(dn, de, pn, pe, seed, kv=5, ke=6, vscale=1.0, escale=1.0):
    rng = np.random.default_rng(seed)
    ends = lambda n, m: rng.integers(0, n, size=m).astype(np.uint64)  # noqa: E731
    d = Graph(vscale * rng.normal(size=(dn, kv)), escale * rng.normal(size=(de, ke)), ends(dn, de), ends(dn, de))
    p = Graph(vscale * rng.normal(size=(pn, kv)), escale * rng.normal(size=(pe, ke)), ends(pn, pe), ends(pn, pe))
    return d, p


def _check(d, p, iters, **kw):
    ref = kernel_algebra.match(d, p, iters, **kw)
    mu = matcher.match(d, p, "fp64", num_iters=iters, **kw)
    assert np.isfinite(mu).all()
    assert np.abs(mu - ref).max() <= REL * max(1.0, np.abs(ref).max())


# lanes, warps of a group, columns and pattern vertices of a lane; ragged last
# stages (two vertices each), more groups than vertices
@pytest.mark.parametrize("pn,pe", [(1, 1), (31, 32), (33, 31), (32, 33), (64, 64), (65, 20), (20, 65),
                                   (128, 128), (64, 129), (128, 255), (5, 256)])
@pytest.mark.parametrize("dn", [1, 5001])
def test_vertex_shapes(cuda, dn, pn, pe):
    d, p = _graphs(dn, 3 * dn + 2, pn, pe, seed=pn * 1000 + pe)
    _check(d, p, 3)


# constants beyond 2^13: the whole launch in FP64 (distances of thousands); and
# below it with some vertices and edges far outside: their stages in FP64
@pytest.mark.parametrize("vscale,escale", [(4e3, 1.0), (1.0, 4e3), (3e4, 3e4), (1e-9, 1e-9), (1e9, 1e9)])
def test_scales(cuda, vscale, escale):
    d, p = _graphs(700, 2500, 7, 12, seed=4, vscale=vscale, escale=escale)
    _check(d, p, 3)


@pytest.mark.parametrize("far", [2e3, 1e5, 1e12])
@pytest.mark.parametrize("pn,pe", [(7, 12), (40, 100)])
def test_outliers(cuda, far, pn, pe):
    d, p = _graphs(3000, 9000, pn, pe, seed=9)
    d.edge_feats[::500] *= far
    d.node_feats[::333] *= 3.0
    _check(d, p, 3)


# edges whose costs agree to eps (0: exactly) around each vertex, so that the
# edge maxima's intervals overlap and FP64 decides
@pytest.mark.parametrize("eps", [0.0, 1e-15, 1e-9, 1e-5])
@pytest.mark.parametrize("pn,pe", [(4, 5), (9, 33), (20, 70)])
def test_near_ties(cuda, eps, pn, pe):
    d, p = _graphs(300, 6000, pn, pe, seed=2)
    rng = np.random.default_rng(3)
    d.edge_feats[:] = d.edge_feats[rng.integers(0, 3, size=6000)] + eps * rng.normal(size=(6000, 6))
    d.node_feats[:] = d.node_feats[rng.integers(0, 2, size=300)]
    _check(d, p, 4)


# hubs: in- and out-edges in many chunks, whose partial rows a block combines
@pytest.mark.parametrize("de", [3000, 60001])
@pytest.mark.parametrize("pn,pe", [(5, 9), (30, 64), (10, 130)])
def test_hub_chunks(cuda, de, pn, pe):
    d, p = _graphs(50, de, pn, pe, seed=7)
    d.dsts[: de // 2] = 3
    d.srcs[de // 3:] = 11
    _check(d, p, 3)


# zero BP iterations: mu is the normalised vertex cost matrix itself; with one,
# the edge matrix too.  Feature counts at and past the kernels' widths, odd
# columns, rows shared by data and pattern (distance 0), near pairs.
@pytest.mark.parametrize("kv,ke", [(1, 2), (2, 1), (3, 32), (13, 17), (32, 31), (33, 40)])
@pytest.mark.parametrize("pn,pe", [(1, 2), (7, 13), (65, 66)])
def test_cost_matrices(cuda, kv, ke, pn, pe):
    if kv > 32 and pn == 1:
        pytest.skip("one pattern vertex with more than 32 features has never been taken")
    d, p = _graphs(700, 1100, pn, pe, seed=kv * 100 + ke, kv=kv, ke=ke)
    d.node_feats[5] = p.node_feats[0]
    d.edge_feats[9] = p.edge_feats[0]
    d.edge_feats[11] = p.edge_feats[0] + 1e-9
    _check(d, p, 0)
    _check(d, p, 1)


# rows and patterns outside the fixed-point range of the block's first rows
@pytest.mark.parametrize("far", [50.0, 1e6, 1e200])
def test_cost_matrix_outliers(cuda, far):
    d, p = _graphs(2000, 5000, 6, 11, seed=8)
    d.edge_feats[777] *= far
    d.node_feats[1500] *= min(far, 1e6)
    _check(d, p, 1)
    if far < 1e100:
        p.edge_feats[3] *= far
        _check(d, p, 1)
