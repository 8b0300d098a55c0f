"""Commits on a graph past the one-launch bounds, whose traversals and sweeps run
as captured loops: new least weight, new columns under the same degrees (the
segmented layout is built again into its buffers), new degrees.  Every run after
a commit is the committed graph's; the device-built layout equals the host's."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _csr(n, u, v, w):
    s, d, ww = np.concatenate([u, v]), np.concatenate([v, u]), np.concatenate([w, w])
    order = np.argsort(s.astype(np.int64) * n + d, kind="stable")
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(np.bincount(s, minlength=n))
    arrays = rp.astype(np.int32), d[order].astype(np.int32), ww[order].astype(np.int32)
    return mg.HostGraph.from_csr(*arrays), O.csr_from_arrays(*arrays)


def _check(g, og, src):
    assert np.array_equal(g.bfs(src)[0], O.bfs(og, src))
    want = O.sssp(og, src)[0]
    for direction in (mg.DIR_AUTO, mg.DIR_PULL):
        assert np.array_equal(g.sssp(src, direction=direction)[0], want)
    assert np.array_equal(g.cc()[0], O.cc_minlabel(og))
    for layout in (mg.PR_LAYOUT_SEGMENTED, mg.PR_LAYOUT_GATHER):
        x, info = g.pagerank(mg.PR_TOPOLOGY, tol=1e-6, pr_layout=layout)
        ref, _ = O.pr_norm_f64(og, 0.85, 1e-6, info.iterations)
        assert np.max(np.abs(x - ref)) < 1e-6
    assert mg.selftest_segmented_build(g) > 0
    (lv, sg, _), _ = g.bc(src)
    rlv, rsg, _ = O.bc_f64(og, src)
    assert np.array_equal(lv, rlv) and np.allclose(sg, rsg, rtol=1e-12, atol=0)


def test_commits_with_captured_loops():
    h = mg.HostGraph.rmat(17, 20, seed=43)
    row, col, _ = h.arrays()
    n = h.nv
    src = np.repeat(np.arange(n), np.diff(row))
    up = src < col
    u, v = src[up], col[up].astype(np.int64)
    assert 2 * len(u) > (4 << 20)
    rng = np.random.default_rng(6)
    h0, og0 = _csr(n, u, v, rng.integers(40, 64, len(u)))
    g = mg.Graph(h0)
    _check(g, og0, 0)
    # same structure, smaller weights
    w1 = rng.integers(1, 64, len(u))
    h1, og1 = _csr(n, u, v, w1)
    g.reload(h1)
    _check(g, og1, 0)
    # (a b), (c d) -> (a d), (c b): the same degrees, other columns
    key = set((np.minimum(u, v) * n + np.maximum(u, v)).tolist())
    u2, v2 = u.copy(), v.copy()
    swapped = 0
    for i, j in rng.integers(0, len(u), (4000, 2)).tolist():
        a, b, c, d = u2[i], v2[i], u2[j], v2[j]
        k1, k2 = min(a, d) * n + max(a, d), min(c, b) * n + max(c, b)
        if a == d or c == b or k1 in key or k2 in key or k1 == k2:
            continue
        key -= {min(a, b) * n + max(a, b), min(c, d) * n + max(c, d)}
        key |= {k1, k2}
        v2[i], v2[j] = d, b
        swapped += 1
    assert swapped > 500
    h2, og2 = _csr(n, u2, v2, w1)
    assert np.array_equal(og2.csc_v, og1.csc_v) and not np.array_equal(og2.csc_e, og1.csc_e)
    g.reload(h2)
    _check(g, og2, 1)
    # new degrees
    perm = rng.permutation(n)
    h3, og3 = _csr(n, perm[u], perm[v], w1)
    g.reload(h3)
    _check(g, og3, int(perm[0]))
    g.free()
