"""Weighted PageRank and its adjoint on graphs without heavy rows, closed by the
sweep itself and by the apply kernel (rows averaging up to eight edges and
above): ranks 1e-6 absolute over the sweep count, gradient of random losses
2e-4 relative to its largest element, from the FP64 oracle; the same bits run
after run."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,degree", [(300, 7), (300, 9), (4000, 8), (4000, 40), (70_000, 4), (30_000, 24)])
def test_either_close(n, degree):
    rng = np.random.default_rng(degree)
    m = n * degree // 2
    h = mg.HostGraph.from_entries(n, rng.integers(0, n, m), rng.integers(0, n, m))
    row, col, wt = h.arrays()
    og = O.csr_from_arrays(row, col, wt)
    assert np.max(np.diff(row)) < 128
    g = mg.Graph(h)
    w = (rng.random(og.ne) + 0.05).astype(np.float32)
    loss = rng.standard_normal(og.nv).astype(np.float32)
    got = []
    for ex in (mg.EXEC_GRAPH, mg.EXEC_HOST):
        g.set_float_weights(w)
        x, _ = g.wpagerank(tol=1e-7, exec=ex)
        (grad, lam), _ = g.wpagerank_backward(loss, tol=1e-7, exec=ex)
        got.append((x, grad, lam))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    ref, _ = O.wpr_f64(og, w, 0.85, 1e-12)
    assert np.max(np.abs(x - ref)) < 1e-6
    _, gr, lm = _adjoint(og, w, ref, loss)
    assert np.max(np.abs(lam - lm)) <= 1e-4 * np.max(np.abs(lm))
    assert np.max(np.abs(grad - gr)) <= 2e-4 * np.max(np.abs(gr))
    g.free()
    h.free()


def _adjoint(og, w, x, loss):
    u = np.repeat(np.arange(og.nv), np.diff(og.csc_v))
    w = w.astype(np.float64)
    total = np.bincount(u, w, og.nv)
    p = w / total[u]
    g = loss.astype(np.float64)
    empty = total == 0
    lam = g.copy()
    for _ in range(400):
        t = np.bincount(u, p * lam[og.csc_e], og.nv)
        t[empty] = lam.mean()
        lam = g + 0.85 * t
    t = np.bincount(u, p * lam[og.csc_e], og.nv)
    return p, 0.85 * (x / np.where(empty, 1.0, total))[u] * (lam[og.csc_e] - t[u]), lam
