"""Many traversals whose levels one block runs by itself: each level's count of
new vertices is read by every warp before it is set back, so every vertex of a
level gets its label and gives its place back.  Levels bit-exact with the
oracle, run after run."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(97, 83), (180, 171), (12, 1500)])
def test_every_vertex_of_a_level_is_labelled(rows, cols):
    h = mg.HostGraph.lattice(rows, cols, 0.0, seed=5)
    og = O.csr_from_arrays(*h.arrays())
    assert np.max(np.diff(h.arrays()[0])) < 128
    g = mg.Graph(h)
    for s in (0, og.nv // 2 + cols // 2, og.nv - 1):
        want = O.bfs(og, s)
        for _ in range(40):
            assert np.array_equal(g.bfs(s)[0], want)
    g.free()
    h.free()
