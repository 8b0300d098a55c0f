"""Weighted PageRank and its adjoint over rows at the bounds of the degree
bins and of the heavy-row chunks, with and without relabeling, and the reuse
of the reverse positions across new weights and new columns.  Bounds: 1e-6
max-abs for the forward, 1e-4 normwise relative for the gradient (against the
FP64 adjoint at the same x), the contracts of these entry points."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _graph(hubs, seed):
    rng = np.random.default_rng(seed)
    n = 5000
    src = [rng.integers(0, n, 4 * n)]
    dst = [rng.integers(0, n, 4 * n)]
    for k, d in enumerate(hubs):
        src.append(np.full(d, n + k))
        dst.append(rng.choice(n, d, replace=False))
    return mg.HostGraph.from_entries(n + len(hubs), np.concatenate(src), np.concatenate(dst))


def _check(g, og, seed):
    rng = np.random.default_rng(seed)
    w = rng.uniform(0.05, 1.0, og.ne).astype(np.float32)
    gv = rng.standard_normal(og.nv).astype(np.float32)
    g.set_float_weights(w)
    x, _ = g.wpagerank(tol=1e-7)
    w64 = w.astype(np.float64)
    assert np.max(np.abs(x - O.wpr_f64(og, w64, 0.85, 1e-13)[0])) < 1e-6
    (grad, lam), _ = g.wpagerank_backward(gv, tol=1e-6)
    lam64, gw64, _, _ = O.wpr_adjoint_f64(og, w64, x.astype(np.float64), gv.astype(np.float64), 0.85, 1e-14)
    assert np.max(np.abs(lam - lam64)) / np.max(np.abs(lam64)) < 1e-4
    assert np.max(np.abs(grad - gw64)) / np.max(np.abs(gw64)) < 1e-4


@pytest.mark.parametrize("hubs", [[], [127], [128, 129], [511, 512, 513], [2047, 2048, 2049, 4100]],
                         ids=lambda h: "-".join(map(str, h)) or "none")
def test_row_bounds(hubs):
    h = _graph(hubs, 1 + len(hubs))
    og = O.csr_from_arrays(*h.arrays())
    g = mg.Graph(h)
    _check(g, og, 1)
    _check(g, og, 2)   # new weights on the same columns
    g.free()
    h.free()


def test_new_columns_same_degrees():
    # a relabeled graph (a ring with one hub) whose columns change while every
    # degree stays
    n = 600
    ring = np.arange(n)
    hub = np.full(200, 0)
    a = mg.HostGraph.from_entries(n, np.concatenate([ring, hub]), np.concatenate([(ring + 1) % n, 200 + np.arange(200)]))
    rp, col, _ = a.arrays()
    g = mg.Graph(a)
    _check(g, O.csr_from_arrays(*a.arrays()), 3)
    # exchange the ring neighbours of two degree-2 vertices far apart
    pairs = {(u, v) for u in range(n) for v in col[rp[u]:rp[u + 1]]}
    for (u, v), (x, y) in [((10, 11), (50, 51)), ((450, 451), (500, 501))]:
        for p, q in ((u, v), (v, u), (x, y), (y, x)):
            pairs.discard((p, q))
        for p, q in ((u, x), (x, u), (v, y), (y, v)):
            pairs.add((p, q))
    e = np.array(sorted(pairs), dtype=np.int64)
    assert np.array_equal(np.bincount(e[:, 0], minlength=n), np.diff(rp))
    c = mg.HostGraph.from_csr(rp, e[:, 1].astype(np.int32), np.ones(len(e), np.int32))
    g.reload(c)
    _check(g, O.csr_from_arrays(*c.arrays()), 4)
    g.free()
