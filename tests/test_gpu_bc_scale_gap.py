"""BC with extended path counts on graphs with heavy vertices, where a vertex
has in-neighbours whose counts lie more than 2^1024 apart (a chain of bipartite
layers beside a bare path of the same length): dependencies finite and 1e-5
normwise from the long-double oracle, for one source, several, and a directed
graph's several."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _edges(layers, spokes):
    # source 0, `layers` layers of 4 (count 4^layers); a path of the same length;
    # both end in one vertex, whose neighbours follow; spokes around the source
    w = 4
    lay = 1 + np.arange(layers * w).reshape(layers, w)
    path = 1 + layers * w + np.arange(layers)
    end = 1 + layers * w + layers
    tail = end + 1 + np.arange(5)
    star = tail[-1] + 1 + np.arange(spokes)
    src, dst = [np.zeros(w, int)], [lay[0]]
    for k in range(layers - 1):
        src.append(np.repeat(lay[k], w))
        dst.append(np.tile(lay[k + 1], w))
    src += [[0], path[:-1], lay[-1], [path[-1]], [end], tail[:-1], np.zeros(spokes, int)]
    dst += [[path[0]], path[1:], np.full(w, end), [end], [tail[0]], tail[1:], star]
    return star[-1] + 1, np.concatenate(src), np.concatenate(dst), end


@pytest.mark.parametrize("layers", [40, 255, 300, 520, 800])
@pytest.mark.parametrize("flags", [mg.LOAD_SYM, mg.LOAD_NSYM], ids=["symmetric", "directed"])
def test_counts_far_apart(layers, flags):
    n, src, dst, end = _edges(layers, 300)
    h = mg.HostGraph.from_entries(n, src, dst, flags=flags)
    row, col, wt = h.arrays()
    assert np.max(np.diff(row)) >= 128 or flags == mg.LOAD_NSYM
    og = O.csr_from_arrays(row, col, wt)
    g = mg.Graph(h)
    want = O.bc_ext(og, 0)
    for _ in range(2):   # (the first run starts over with extended counts)
        (lv, sg, dl), _ = g.bc(0)
        assert np.array_equal(lv, want[0])
        assert np.all(np.isfinite(dl))
        if flags == mg.LOAD_SYM:
            assert np.max(np.abs(dl - want[2])) <= 1e-5 * np.max(np.abs(want[2]))
    srcs = [0, int(end), 2]
    got = g.bc_multi(srcs)[0].astype(np.float64)
    assert np.all(np.isfinite(got))
    if flags == mg.LOAD_SYM:
        ref = O.bc_multi_ext(og, srcs)
        assert np.max(np.abs(got - ref)) <= 1e-5 * np.max(np.abs(ref))
    else:
        # over out-edges, level by level, with the oracle's log2 counts
        ref = np.zeros(og.nv)
        u = np.repeat(np.arange(og.nv), np.diff(row))
        for s in srcs:
            l, lg, _ = O.bc_ext(og, s)
            d = np.zeros(og.nv)
            down = (l[u] != O.IUNUSED) & (l[col] == l[u] + 1)
            for x in np.sort(np.unique(l[l != O.IUNUSED]))[::-1]:
                e = np.flatnonzero(down & (l[u] == x))
                np.add.at(d, u[e], np.exp2(lg[u[e]] - lg[col[e]]) * (1.0 + d[col[e]]))
            d[s] = 0.0
            ref += d
        assert np.max(np.abs(got - ref)) <= 1e-5 * np.max(np.abs(ref))
    g.free()
    h.free()
