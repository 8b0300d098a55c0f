"""Push levels over vertices around the heavy-chunk bounds: BFS and SSSP from
the hub and from a leaf of stars whose hub degrees sit at the edges of the
chunk rules, against the oracle (bit-exact)."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deg", [127, 128, 129, 512, 513, 4097, 524288, 524289, 600001])
@pytest.mark.parametrize("direction", [mg.DIR_PUSH, mg.DIR_AUTO, mg.DIR_PULL])
def test_hub_degree(deg, direction):
    # hub 0 with `deg` leaves, every third leaf with a second neighbour, and a
    # second hub over those: two levels of heavy and light vertices
    leaf = np.arange(1, deg + 1)
    third = leaf[::3]
    far = deg + 1 + np.arange(len(third))
    hub2 = deg + 1 + len(third)
    src = np.concatenate([np.zeros(deg, np.int64), third, np.full(len(far), hub2)])
    dst = np.concatenate([leaf, far, far])
    w = np.random.default_rng(deg).integers(1, 65, len(src))
    h = mg.HostGraph.from_entries(hub2 + 1, src, dst, w)
    rp, col, wt = h.arrays()
    og = O.csr_from_arrays(rp, col, wt)
    g = mg.Graph(h)
    for s in (0, deg // 2, og.nv - 1):
        assert np.array_equal(g.bfs(s, direction=direction)[0], O.bfs(og, s))
        assert np.array_equal(g.sssp(s, direction=direction)[0], O.sssp(og, s)[0])
    g.free()
    h.free()


def test_many_sources_of_a_batch():
    # more sources than one round of the init block's threads
    hs = [mg.HostGraph.rmat(6 + i % 3, 8, seed=i + 1) for i in range(300)]
    b = mg.Batch(hs)
    levels, _ = b.bfs([i % hs[i].nv for i in range(300)])
    for i, h in enumerate(hs):
        assert np.array_equal(levels[i], O.bfs(O.csr_from_arrays(*h.arrays()), i % h.nv)), i
    b.free()


@pytest.mark.parametrize("deg", [129, 255, 256, 257, 512, 513, 4097, 40000])
@pytest.mark.parametrize("flags", [mg.LOAD_SYM, mg.LOAD_NSYM], ids=["symmetric", "directed"])
def test_bc_long_entries(deg, flags):
    # BC over entries around the backward sweep's chunk bound: a hub over
    # `deg` middle vertices that reach `deg` // 2 + 1 ends by two edges each,
    # and a second, smaller hub on the way
    mid = 1 + np.arange(deg)
    end = 1 + deg + np.arange(deg // 2 + 1)
    hub2 = 1 + deg + len(end)
    some = end[:300]
    src = np.concatenate([np.zeros(deg, np.int64), mid, mid, [0], np.full(len(some), hub2)])
    dst = np.concatenate([mid, end[(mid - 1) // 2], end[mid % len(end)], [hub2], some])
    h = mg.HostGraph.from_entries(hub2 + 1, src, dst, flags=flags)
    rp, col, _ = h.arrays()
    og = O.csr_from_arrays(*h.arrays())
    g = mg.Graph(h)
    for s in (0, 1, og.nv - 1):
        (lv, sg, dl), _ = g.bc(s)
        want = O.bc_f64(og, s)
        assert np.array_equal(lv, want[0]) and np.array_equal(sg, want[1])
        u = np.repeat(np.arange(og.nv), np.diff(rp))
        ref = np.zeros(og.nv)
        for at in range(int(lv[lv < 0x64646464].max()) - 1, -1, -1):
            e = (lv[u] == at) & (lv[col] == at + 1)
            np.add.at(ref, u[e], sg[u[e]] * (1.0 + ref[col[e]]) / sg[col[e]])
        assert np.max(np.abs(dl - ref)) <= 1e-5 * max(1.0, np.max(np.abs(ref)))
    g.free()
    h.free()


@pytest.mark.parametrize("direction", [mg.DIR_AUTO, mg.DIR_PULL])
def test_sssp_large_weights(direction):
    # three layers, edges forward only: every path's sum is in range, an
    # unreached vertex's label plus a weight would wrap
    rng = np.random.default_rng(12)
    a, b, c = np.arange(300), np.arange(300, 700), np.arange(700, 1000)
    src = np.concatenate([rng.choice(a, 4000), rng.choice(b, 4000)])
    dst = np.concatenate([rng.choice(b, 4000), rng.choice(c, 4000)])
    wt = rng.integers(500_000_000, 800_000_000, 8000)
    h = mg.HostGraph.from_entries(1000, src, dst, wt, flags=mg.LOAD_NSYM)
    og = O.csr_from_arrays(*h.arrays())
    src = np.repeat(np.arange(og.nv), np.diff(og.csc_v))
    g = mg.Graph(h)
    for s in (0, 7, 400, og.nv - 1):
        far = np.full(og.nv, 1 << 40)
        far[s] = 0
        for _ in range(2):
            np.minimum.at(far, og.csc_e, far[src] + og.csc_ev)
        expect = np.where(far < 1 << 40, far, 1684300900)
        assert far[far < 1 << 40].max() < 1684300900
        for exec_ in (mg.EXEC_GRAPH, mg.EXEC_HOST):
            assert np.array_equal(g.sssp(s, direction=direction, exec=exec_)[0], expect)
    g.free()
    h.free()
