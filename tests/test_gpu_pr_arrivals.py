"""One-launch PageRank over so many sweeps that the arrivals of a long row's
chunks add up to more than 2^31: a star of 3.1 M spokes (12,158 chunks of the
hub's row) at damping 1, where the mass swings between hub and spokes for ever
and every sweep's L1 change is the same to the last bit."""
import ctypes as C

import numpy as np
import pytest

import multigraph_gb300 as mg

pytestmark = pytest.mark.gpu


def _residual(g, sweeps):
    o = g._opts(None, dict(damping=1.0, tol=1e-6, max_iter=sweeps))
    info = mg.RunInfo()
    st = mg.lib.mg_pagerank(g._h, mg.PR_TOPOLOGY, C.byref(o), None, C.byref(info))
    assert st == mg.MG_ERR_ITER_LIMIT and info.iterations == sweeps
    return info.residual


def test_more_arrivals_than_a_counter_holds():
    spokes = 3_112_448
    h = mg.HostGraph.from_entries(spokes + 1, np.zeros(spokes, np.int32), 1 + np.arange(spokes))
    assert h.ne <= 6 << 20
    g = mg.Graph(h)
    h.free()
    want = _residual(g, 50)
    assert 1.0 < want <= 2.001
    chunks = -(-spokes // 256)
    got = _residual(g, 2**31 // chunks + 5)
    assert abs(got - want) <= 1e-9, (got, want)
    g.free()
