"""Directed graphs without a vertex of 128 out-edges but with a long in-row
(which relabels nothing): path counts there are not summed over the whole
in-row by one thread, on either side of the bound (127 / 128 in-edges).
Levels and path counts equal to the oracle's; dependencies 1e-5 normwise; a
pull row of two million edges costs under a millisecond (220 where one thread
walks it)."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _graph(spokes):
    # a path of 60 vertices whose 5th and 40th also point at the hub, the hub
    # at the path's last vertex; every spoke points at the hub
    path = np.arange(60)
    hub, first = 60, 61
    src = [path[:-1], [5, 40], [hub], first + np.arange(spokes)]
    dst = [path[1:], [hub, hub], [59], np.full(spokes, hub)]
    return mg.HostGraph.from_entries(first + spokes, np.concatenate(src), np.concatenate(dst), flags=mg.LOAD_NSYM)


@pytest.mark.parametrize("spokes", [124, 125, 126, 127, 3000, 2_000_000])
def test_bc_reaches_an_in_hub(spokes):
    h = _graph(spokes)
    row, col, _ = h.arrays()
    og = O.csr_from_arrays(*h.arrays())
    assert np.max(np.diff(row)) < 128
    g = mg.Graph(h)
    want = O.bc_f64(og, 0)
    lv = want[0]
    delta = np.zeros(og.nv)
    for u in np.argsort(lv[:61], kind="stable")[::-1]:   # (spokes are not reached from 0)
        for v in col[row[u]:row[u + 1]]:
            if lv[u] != O.IUNUSED and lv[v] == lv[u] + 1:
                delta[u] += want[1][u] * (1.0 + delta[v]) / want[1][v]
    for ex in (mg.EXEC_GRAPH, mg.EXEC_HOST):
        g.bc(0, exec=ex)
        (glv, sg, dl), info = g.bc(0, exec=ex)
        assert np.array_equal(glv, lv) and np.array_equal(sg, want[1])
        assert np.max(np.abs(dl - delta)) <= 1e-5 * np.max(np.abs(delta))
        assert info.device_ms < 50.0, info.device_ms
    g.free()
    h.free()
