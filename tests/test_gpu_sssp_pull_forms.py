"""SSSP with every level pulled (offers past the frontier bitmap's test), with
the direction switch (every reached neighbour's offer) and pushed, in turn on
one graph past the one-launch bound and one below it, as captured loops and
host loops: distances equal to the oracle's, also where most vertices stay
unreached and where weights are large."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _random(n, degree, parts, wmax, seed):
    # `parts` random graphs apart
    rng = np.random.default_rng(seed)
    m = n * degree // 2
    part = rng.integers(0, parts, m)
    k = n // parts
    return mg.HostGraph.from_entries(n, part * k + rng.integers(0, k, m), part * k + rng.integers(0, k, m),
                                     rng.integers(1, wmax + 1, m))


@pytest.mark.parametrize("kind", ["rmat17", "rmat13", "random", "parts", "large weights"])
def test_forms_in_turn(kind):
    if kind.startswith("rmat"):
        h = mg.HostGraph.rmat(int(kind[4:]), 16, seed=4)
    elif kind == "random":
        h = _random(200_000, 20, 1, 64, 1)
    elif kind == "parts":
        h = _random(400_000, 12, 7, 64, 2)
    else:
        h = _random(150_000, 24, 1, 90_000_000, 3)   # a dozen steps stay below UNSET = 0x64646464
    og = O.csr_from_arrays(*h.arrays())
    g = mg.Graph(h)
    for src in (0, og.nv - 1):
        want = O.sssp(og, src)[0]
        for _ in range(2):
            for direction in (mg.DIR_PULL, mg.DIR_AUTO, mg.DIR_PUSH):
                for ex in (mg.EXEC_GRAPH, mg.EXEC_HOST):
                    assert np.array_equal(g.sssp(src, direction=direction, exec=ex)[0], want), (direction, ex)
    g.free()
    h.free()
