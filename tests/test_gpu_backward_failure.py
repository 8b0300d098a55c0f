"""The BC backward sweeps' own barrier failure: a host-driven, pull-only forward
traversal has no grid barrier, so under injection the backward sweep is the one
whose bounded wait runs out.  It ends with MG_ERR_CUDA naming the backward
kernel, on graphs with and without heavy vertices, and the next run is right."""
import os

import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["path", "hub"])
def test_backward_barrier_timeout(kind):
    if kind == "path":
        h = mg.HostGraph.from_entries(400, np.arange(399), np.arange(1, 400))
    else:
        h = mg.HostGraph.rmat(11, 16, seed=5)
        assert np.max(np.diff(h.arrays()[0])) >= 300   # long entries, too
    og = O.csr_from_arrays(*h.arrays())
    g = mg.Graph(h)
    for _ in range(2):
        os.environ["MG_FAIL_BARRIER"] = "1"
        try:
            with pytest.raises(mg.MGError) as e:
                g.bc(3, direction=mg.DIR_PULL, exec=mg.EXEC_HOST)
        finally:
            del os.environ["MG_FAIL_BARRIER"]
        assert e.value.status == mg.MG_ERR_CUDA
        assert "backward" in str(e.value)
        for ex in (mg.EXEC_HOST, mg.EXEC_GRAPH):
            (lv, sg, dl), _ = g.bc(3, direction=mg.DIR_PULL, exec=ex)
            rlv, rsg, rdl = O.bc_f64(og, 3)
            assert np.array_equal(lv, rlv) and np.array_equal(sg, rsg)
            assert np.max(np.abs(dl - rdl)) <= 1e-5 * max(1.0, np.max(np.abs(rdl)))
    g.free()
    h.free()
