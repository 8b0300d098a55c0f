"""The segmented PageRank layout's windows of 32 rows -- sorted ones, ones of
more than 512 pieces, ones with a warp row (more than 32 pieces), the last
one of a row count off 32, a layout with a tail -- against the FP64 oracle for
the same sweeps (1e-6 max-abs, the contract); and the layout that the device
builds against the host's."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _make(kind):
    rng = np.random.default_rng(8)
    n = 57344 * 2 + 37
    deg = rng.integers(0, 6, n)
    if kind == "long":          # 32 rows of ~22 pieces each: above 512 in a window, no warp row
        deg[64:96] = 700
    elif kind == "edge":        # 32 rows of 15 to 17 pieces each: at the bound of 512
        deg[64:96] = 500
    elif kind == "warp":        # a warp row in a window of short rows
        deg[64] = 1500
    elif kind == "rows":        # rows at the bounds of the build's subs, and far above them
        deg[[5, 70, 71, 72, 73, 900, 5000]] = [2047, 2048, 2049, 4096, 4097, 40000, 90001]
    elif kind == "tail":        # more vertices than the segments hold
        n = 57344 * 64 + 37
        deg = rng.integers(0, 2, n)
    src = np.repeat(np.arange(n, dtype=np.int64), deg)
    if kind == "tail":
        dst = np.where(rng.random(len(src)) < 0.7, rng.integers(0, 57344 * 60, len(src)), rng.integers(0, n, len(src)))
    else:
        dst = rng.integers(0, n, len(src))
    src, dst = np.concatenate([src, np.arange(n - 1)]), np.concatenate([dst, np.arange(1, n)])
    return mg.HostGraph.from_entries(n, src, dst)


@pytest.mark.parametrize("kind", ["short", "long", "edge", "warp", "rows", "tail"])
def test_windows(kind):
    h = _make(kind)
    og = O.csr_from_arrays(*h.arrays())
    g = mg.Graph(h)
    ref = None
    for exec_ in (mg.EXEC_GRAPH, mg.EXEC_HOST):
        x, info = g.pagerank(mg.PR_TOPOLOGY, tol=1e-4, exec=exec_, pr_layout=mg.PR_LAYOUT_SEGMENTED)
        if ref is None:
            ref, _ = O.pr_norm_f64(og, 0.85, 0.0, info.iterations)
        assert np.max(np.abs(x.astype(np.float64) - ref)) < 1e-6
    g.free()
    h.free()


@pytest.mark.parametrize("kind", ["short", "long", "edge", "warp", "rows", "tail", "directed", "small"])
def test_device_build(kind):
    # the layout built on the device, byte for byte the host's
    if kind == "directed":
        rng = np.random.default_rng(4)
        s = np.concatenate([rng.integers(0, 90000, 400000), rng.integers(0, 90000, 5000), np.full(7000, 3)])
        d = np.concatenate([rng.integers(0, 90000, 400000), np.full(5000, 77), rng.integers(0, 90000, 7000)])
        h = mg.HostGraph.from_entries(90000, s, d, flags=mg.LOAD_NSYM)
    elif kind == "small":
        h = mg.HostGraph.rmat(7, 4, seed=2)
    else:
        h = _make(kind)
    g = mg.Graph(h)
    assert mg.selftest_segmented_build(g) > 0
    g.free()
    h.free()
