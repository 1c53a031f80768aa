"""FP32 patterns wider than 64 edges with few vertices: both forms of the vertex phase
at the graph sizes between which the plan chooses, against the numpy model.

Tolerance: that of test_gpu_hub_patterns.py (a vertex's sum is a hub's here)."""
import numpy as np
import pytest

import kernel_algebra
from application_classification_gb300 import matcher
from test_gpu_fp64_integer import _graphs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pn,pe,dn", [(1, 70, 65535), (1, 70, 65536), (2, 128, 65536), (8, 132, 32767),
                                      (8, 132, 32768), (8, 256, 32768), (9, 132, 65535), (9, 132, 65536),
                                      (16, 168, 65536), (17, 168, 65536)])
def test_few_vertices(cuda, pn, pe, dn):
    d, p = _graphs(dn, dn + 1, pn, pe, seed=pn + pe)
    ref = kernel_algebra.match(d, p, 2)
    mu = matcher.match(d, p, "mixed", num_iters=2)
    degree = np.bincount(np.concatenate([p.srcs, p.dsts]).astype(int)).max()
    assert np.abs(mu - ref).max() <= max(1e-4, degree * 60 * 2.0**-24)
