"""Personalised PageRank at the bounds of its pass widths (1-4, 5-8, 9-16,
17-32 seeds, a remainder pass) and of its heavy-row split (256 in-edges),
with and without dangling vertices, against the FP64 oracle for the same
sweeps (max-abs 1e-6, the contract of every PageRank result here)."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _stars():
    # hubs of 255, 256, 257, 512, 513 and 2400 in-edges over shared leaves
    src, dst = [], []
    for k, d in enumerate([255, 256, 257, 512, 513, 2400]):
        src.append(np.full(d, k))
        dst.append(6 + np.arange(d))
    return mg.HostGraph.from_entries(2406, np.concatenate(src), np.concatenate(dst))


def _directed():
    # vertices 400.. have in-edges only: dangling
    rng = np.random.default_rng(5)
    s = rng.integers(0, 400, 6000)
    d = rng.integers(0, 700, 6000)
    return mg.HostGraph.from_entries(700, s, d, flags=mg.LOAD_NSYM)


@pytest.mark.parametrize("make", [_stars, _directed, lambda: mg.HostGraph.lattice(37, 41, 0.05, seed=2)],
                         ids=["stars", "directed", "lattice"])
@pytest.mark.parametrize("count", [1, 4, 5, 8, 9, 16, 17, 32, 33, 45])
def test_pass_widths(make, count):
    h = make()
    og = O.csr_from_arrays(*h.arrays())
    g = mg.Graph(h)
    seeds = (np.arange(count) * 53) % og.nv
    seeds[count // 2] = seeds[0]   # a seed twice
    x, _ = g.ppr_batch(seeds, tol=1e-6)
    for k0 in range(0, count, 32):
        part = seeds[k0:k0 + 32]
        alone, info = g.ppr_batch(part, tol=1e-6)
        assert np.array_equal(alone, x[k0:k0 + 32])
        for i in {0, len(part) // 2, len(part) - 1}:
            ref, _ = O.ppr_f64(og, int(part[i]), 0.85, 0.0, info.iterations)
            assert np.max(np.abs(x[k0 + i].astype(np.float64) - ref)) < 1e-6
    g.free()
    h.free()
