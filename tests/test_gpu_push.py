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
