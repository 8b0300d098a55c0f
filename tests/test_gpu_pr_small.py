"""PageRank's one-launch form (small graphs, default layout) at the bounds of
its row classes -- 15/16 edges, 255..257 and 512/513 edges, a single vertex,
dangling vertices, directed hubs -- against the FP64 oracle for the same
sweeps (1e-6 max-abs, the contract), and the iteration cap and the barrier's
error path."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _make(kind):
    rng = np.random.default_rng(3)
    if kind == "rows":          # hubs around every bound over a sparse base
        n = 3000
        src = [rng.integers(0, n, 3 * n)]
        dst = [rng.integers(0, n, 3 * n)]
        for k, d in enumerate([7, 8, 15, 16, 31, 32, 33, 127, 128, 129, 255, 256, 257, 511, 512, 513, 2900]):
            src.append(np.full(d, n + k))
            dst.append(rng.choice(n, d, replace=False))
        return mg.HostGraph.from_entries(n + 17, np.concatenate(src), np.concatenate(dst))
    if kind == "directed":      # in-hubs of 300 and 600, dangling vertices
        s = np.concatenate([rng.integers(0, 900, 4000), rng.choice(900, 300, replace=False), rng.choice(900, 600, replace=False)])
        d = np.concatenate([rng.integers(0, 1200, 4000), np.full(300, 1000), np.full(600, 1001)])
        return mg.HostGraph.from_entries(1200, s, d, flags=mg.LOAD_NSYM)
    if kind == "one":
        return mg.HostGraph.from_csr([0, 0], [])
    if kind == "star":
        return mg.HostGraph.from_entries(20001, np.zeros(20000, np.int64), 1 + np.arange(20000))
    if kind == "lattice":
        return mg.HostGraph.lattice(61, 53, 0.05, seed=4)
    return mg.HostGraph.rmat(12, 16, seed=6)


@pytest.mark.parametrize("kind", ["rows", "directed", "one", "star", "lattice", "rmat"])
def test_rows(kind):
    h = _make(kind)
    og = O.csr_from_arrays(*h.arrays())
    g = mg.Graph(h)
    for tol in (1e-4, 1e-6):
        x, info = g.pagerank(mg.PR_TOPOLOGY, tol=tol)
        ref, _ = O.pr_norm_f64(og, 0.85, 0.0, info.iterations)
        assert np.max(np.abs(x.astype(np.float64) - ref)) < 1e-6
        # the host-driven loop runs the other kernels: the same sweeps
        y, other = g.pagerank(mg.PR_TOPOLOGY, tol=tol, exec=mg.EXEC_HOST)
        assert abs(info.iterations - other.iterations) <= 1
    g.free()
    h.free()


def test_iteration_cap():
    h = _make("rmat")
    g = mg.Graph(h)
    with pytest.raises(mg.MGError) as e:
        g.pagerank(mg.PR_TOPOLOGY, tol=1e-6, max_iter=3)
    assert e.value.status == mg.MG_ERR_ITER_LIMIT
    assert g.pagerank(mg.PR_TOPOLOGY, tol=1e-6)[1].iterations > 3
    g.free()


def test_barrier_timeout_reports(monkeypatch):
    h = _make("rmat")
    g = mg.Graph(h)
    want, _ = g.pagerank(mg.PR_TOPOLOGY, tol=1e-6)
    monkeypatch.setenv("MG_FAIL_BARRIER", "1")
    with pytest.raises(mg.MGError) as e:
        g.pagerank(mg.PR_TOPOLOGY, tol=1e-6)
    assert e.value.status == mg.MG_ERR_CUDA
    monkeypatch.delenv("MG_FAIL_BARRIER")
    assert np.array_equal(g.pagerank(mg.PR_TOPOLOGY, tol=1e-6)[0], want)
    g.free()
