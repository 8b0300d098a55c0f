"""Components of graphs that strain the hub-first linking: long paths beside a
hub (chains of every length under the first link), many small components, a
hub whose leaves are hubs of other trees, in ascending, descending and
shuffled numbering; labels bit-exact against the oracle."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _edges(kind):
    if kind == "path_hub":      # a path of 150 K and a hub of 200 leaves, apart
        p = np.arange(150_000)
        return np.concatenate([p[:-1], np.full(200, 150_000)]), np.concatenate([p[1:], 150_001 + np.arange(200)])
    if kind == "comb":          # a hub at the end of each of 40 paths of 999, joined in a chain of hubs
        src, dst = [], []
        for k in range(40):
            base = k * 1200
            src.append(base + np.arange(998))
            dst.append(base + 1 + np.arange(998))
            src.append(np.full(150, base + 998))
            dst.append(base + 999 + np.arange(150))
            if k:
                src.append([base])
                dst.append([base - 1200 + 999])
        return np.concatenate(src), np.concatenate(dst)
    if kind == "pairs":         # 30,000 pairs and one star
        a = np.arange(30_000) * 2
        return np.concatenate([a, np.full(300, 60_000)]), np.concatenate([a + 1, 60_001 + np.arange(300)])
    rng = np.random.default_rng(4)   # hubs sharing leaves, sparse
    return rng.integers(0, 300, 40_000), rng.integers(300, 60_000, 40_000)


@pytest.mark.parametrize("kind", ["path_hub", "comb", "pairs", "hubs"])
@pytest.mark.parametrize("order", ["up", "down", "shuffled"])
def test_components(kind, order):
    src, dst = _edges(kind)
    n = int(max(src.max(), dst.max())) + 1
    perm = np.arange(n) if order == "up" else np.arange(n)[::-1] if order == "down" else \
        np.random.default_rng(1).permutation(n)
    h = mg.HostGraph.from_entries(n, perm[src], perm[dst])
    g = mg.Graph(h)
    want = O.cc_minlabel(O.csr_from_arrays(*h.arrays()))
    for _ in range(3):
        assert np.array_equal(g.cc()[0], want)
    g.free()
    h.free()
