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


# large enough for a batch to combine the statistics beside the edge phase: a
# pattern that forms a group of its own has the bits of its single match, on the
# first call (captured), on the relaunch, and on another stream; and single plans
# give the same bits with two matches in flight and with phase timing
@pytest.mark.parametrize("precision,pn,pe", [("mixed", 16, 60), ("mixed", 20, 90), ("fp64", 16, 60)])
def test_statistics_beside_edge_phase(cuda, precision, pn, pe):
    import torch

    d, p, _ = graph.workload(f"rmat16_{pn}_{pe}")
    data = matcher.DataGraph(d)
    want = matcher.Plan(data, p, precision, kernel_timing=True).run()
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    plans = [matcher.Plan(data, p, precision) for _ in range(2)]
    outs = []
    for plan, st in zip(plans * 2, streams * 2):
        with torch.cuda.stream(st):
            outs.append(plan.run(stream=st))
    batch = matcher.Batch(data, [p, p], precision)
    for st in (streams[0], streams[0], streams[1]):
        with torch.cuda.stream(st):
            outs += [o.clone() for o in batch.run(stream=st)]
        st.synchronize()
    torch.cuda.synchronize()
    for o in outs:
        assert torch.equal(o, want)
