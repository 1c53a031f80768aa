"""FP32 vertex phase of patterns wider than 64 edges (rows of one or two warps), and
the statistics combined beside the next edge phase on a plan's own stream.

Tolerance: the mixed path's 1e-4 absolute (test_gpu_parity.py) after two
iterations, before FP32 rounding is amplified through a column's normaliser."""
import numpy as np
import pytest

import kernel_algebra
from application_classification_gb300 import graph, matcher
from test_gpu_fp64_integer import _graphs

pytestmark = pytest.mark.gpu


# padded columns at each count of rows per block (15 ... 4), one and two warps a
# row; more rows than vertices; two pattern vertices a lane
@pytest.mark.parametrize("pn,pe", [(5, 65), (33, 72), (64, 100), (20, 128), (128, 129), (40, 150),
                                   (70, 170), (30, 204), (128, 256)])
@pytest.mark.parametrize("dn", [3, 4001])
def test_wide_vertex_phase(cuda, dn, pn, pe):
    d, p = _graphs(dn, 3 * dn + 2, pn, pe, seed=pn * 1000 + pe)
    ref = kernel_algebra.match(d, p, 2)
    mu = matcher.match(d, p, "mixed", num_iters=2)
    assert np.abs(mu - ref).max() <= 1e-4


# large enough for the statistics to run beside the edge phase: the same bits on
# another stream, on a reused plan, with two plans' matches in flight, and with
# phase timing (statistics in line)
@pytest.mark.parametrize("precision,pn,pe", [("mixed", 16, 32), ("mixed", 20, 90), ("fp64", 16, 32)])
def test_side_stream(cuda, precision, pn, pe):
    import torch

    d, p, _ = graph.workload(f"rmat16_{pn}_{pe}")
    data = matcher.DataGraph(d)
    plans = [matcher.Plan(data, p, precision) for _ in range(2)]
    timed = matcher.Plan(data, p, precision, kernel_timing=True)
    want = timed.run()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = []
    for _ in range(2):
        for plan, st in zip(plans, streams):
            with torch.cuda.stream(st):
                outs.append(plan.run(stream=st))
    torch.cuda.synchronize()
    for o in outs:
        assert torch.equal(o, want)
