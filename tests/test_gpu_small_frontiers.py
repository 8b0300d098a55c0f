"""Traversals whose levels one block runs by itself (graphs without vertices
of 128 edges, small frontiers): frontiers crossing the hand-over bounds both
ways, more levels than one block phase holds, directed graphs (path counts
pulled over in-edges), several components.  BFS and BC levels bit-exact, path
counts within FP64 rounding of the oracle, dependencies 1e-5 relative."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _edges(kind):
    if kind == "path":            # 25,000 levels of one vertex
        v = np.arange(25_000)
        return v[:-1], v[1:]
    if kind == "ladder":          # 3 x 3,000
        v = np.arange(9_000).reshape(3, 3_000)
        return (np.concatenate([v[:, :-1].ravel(), v[:-1].ravel()]), np.concatenate([v[:, 1:].ravel(), v[1:].ravel()]))
    if kind == "diamonds":        # frontiers 1, 3, 9, .. 6561 and back, twice
        src, dst, base, layer = [], [], 0, np.array([0])
        nxt = 1
        for w in [3, 9, 27, 81, 243, 729, 2187, 6561, 2187, 729, 243, 81, 27, 9, 3, 1] * 2:
            new = nxt + np.arange(w)
            nxt += w
            k = max(w, len(layer))
            src.append(layer[np.arange(k) * len(layer) // k])
            dst.append(new[np.arange(k) * w // k])
            layer = new
        return np.concatenate(src), np.concatenate(dst)
    if kind == "wide":            # levels of 380..515 vertices: rungs of four columns, width drifting over the bounds
        src, dst, nxt, layer = [], [], 1, np.zeros(1, np.int64)
        for k in range(60):
            w = 380 + (k * 37) % 136
            new = nxt + np.arange(w)
            nxt += w
            for s in range(3):
                src.append(layer[(np.arange(w) + s) % len(layer)] if len(layer) > 1 else layer[np.zeros(w, int)][: min(w, 100)])
                dst.append(new if len(layer) > 1 else new[: min(w, 100)])
            layer = new
        return np.concatenate(src), np.concatenate(dst)
    v = np.arange(40 * 30).reshape(40, 30)   # two lattices apart
    a = np.concatenate([v[:, :-1].ravel(), v[:-1].ravel()])
    b = np.concatenate([v[:, 1:].ravel(), v[1:].ravel()])
    return np.concatenate([a, a + 1200]), np.concatenate([b, b + 1200])


def _delta(row, col, lv, sg):
    """FP64 dependencies over out-edges, level by level."""
    u = np.repeat(np.arange(len(row) - 1), np.diff(row))
    down = (lv[u] != 0x64646464) & (lv[col] == lv[u] + 1)
    u, w = u[down], col[down]
    by = np.argsort(lv[u], kind="stable")[::-1]
    u, w = u[by], w[by]
    cut = np.flatnonzero(np.diff(lv[u])) + 1
    d = np.zeros(len(row) - 1)
    for a, b in zip(np.concatenate([[0], cut]), np.concatenate([cut, [len(u)]])):
        if b > a:
            np.add.at(d, u[a:b], sg[u[a:b]] * (1.0 + d[w[a:b]]) / sg[w[a:b]])
    return d


@pytest.mark.parametrize("kind", ["path", "ladder", "diamonds", "wide", "two"])
@pytest.mark.parametrize("flags", [mg.LOAD_SYM, mg.LOAD_NSYM], ids=["symmetric", "directed"])
def test_levels(kind, flags):
    src, dst = _edges(kind)
    n = int(max(src.max(), dst.max())) + 1
    h = mg.HostGraph.from_entries(n, src, dst, flags=flags)
    og = O.csr_from_arrays(*h.arrays())
    assert np.max(np.diff(h.arrays()[0])) < 128
    g = mg.Graph(h)
    for s in {0, og.nv // 2, og.nv - 1}:
        for ex in (mg.EXEC_GRAPH, mg.EXEC_HOST):
            assert np.array_equal(g.bfs(s, exec=ex)[0], O.bfs(og, s))
        assert np.array_equal(g.bfs(s, direction=mg.DIR_PUSH)[0], O.bfs(og, s))
    for s in {0, og.nv // 2}:
        (lv, sg, dl), _ = g.bc(s)
        want = O.bc_f64(og, s)
        assert np.array_equal(lv, want[0])
        assert np.allclose(sg, want[1], rtol=1e-12, atol=0)
        ref = _delta(*h.arrays()[:2], lv, sg)
        if flags == mg.LOAD_SYM:   # (the oracle's dependencies, as the reference's, take the graph as symmetric)
            assert np.allclose(ref, want[2], rtol=1e-9, atol=1e-9)
        assert np.max(np.abs(dl - ref)) <= 1e-5 * max(1.0, np.max(np.abs(ref)))
    g.free()
    h.free()
