"""Batched BC over the forms of its path counts (32-bit integers, FP64,
extended) and around the mask-free levels' bounds (rows of 255..513 edges,
groups of 1..33 sources), against the FP64 (long-double where counts pass
FP64's comfort) oracle: 1e-5 normwise, the contract of BC scores here."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _layers(count, width=30):
    # complete bipartite between neighbouring layers: width^k shortest paths
    a = np.arange(width)
    src, dst = [], []
    for k in range(count - 1):
        src.append(np.repeat(k * width + a, width))
        dst.append(np.tile((k + 1) * width + a, width))
    return mg.HostGraph.from_entries(count * width, np.concatenate(src), np.concatenate(dst))


def _check(g, og, src, ext=False, **kw):
    got = g.bc_multi(src, **kw)[0].astype(np.float64)
    ref = O.bc_multi_ext(og, src) if ext else O.bc_multi_f64(og, src)
    assert np.max(np.abs(got - ref)) / np.max(np.abs(ref)) < 1e-5


@pytest.mark.parametrize("layers", [3, 5, 6, 7, 8, 19, 24])   # 30^5 < 2^29 < 30^6; 30^18 < 2^90 < 30^19
def test_count_forms(layers):
    h = _layers(layers)
    og = O.csr_from_arrays(*h.arrays())
    g = mg.Graph(h)
    src = [0, 1, og.nv - 1, og.nv // 2, 7, 7]
    _check(g, og, src, ext=layers > 19)
    _check(g, og, [0], ext=layers > 19)   # (the graph keeps the form it reached)
    g.free()
    h.free()


@pytest.mark.parametrize("count", [1, 5, 32, 33])
@pytest.mark.parametrize("direction", [mg.DIR_AUTO, mg.DIR_PULL, mg.DIR_PUSH])
def test_row_bounds(count, direction):
    rng = np.random.default_rng(8)
    n = 3000
    src = [rng.integers(0, n, 12 * n)]
    dst = [rng.integers(0, n, 12 * n)]
    for k, d in enumerate([255, 256, 257, 512, 513, 2100]):
        src.append(np.full(d, n + k))
        dst.append(rng.choice(n, d, replace=False))
    h = mg.HostGraph.from_entries(n + 6, np.concatenate(src), np.concatenate(dst))
    og = O.csr_from_arrays(*h.arrays())
    g = mg.Graph(h)
    _check(g, og, (np.arange(count) * 97) % og.nv, direction=direction)
    g.free()
    h.free()


@pytest.mark.parametrize("count", [1, 4, 5, 31, 33])
@pytest.mark.parametrize("direction", [mg.DIR_AUTO, mg.DIR_PULL, mg.DIR_PUSH])
def test_low_degree_rows(count, direction):
    # a lattice with hubs of 8..127 edges (rows past the thread path) and a
    # second component; sources close together, so rows meet many at a level
    rng = np.random.default_rng(9)
    v = np.arange(70 * 60).reshape(70, 60)
    src = [v[:, :-1].ravel(), v[:-1].ravel()]
    dst = [v[:, 1:].ravel(), v[1:].ravel()]
    n = v.size
    for k, d in enumerate([8, 9, 31, 32, 33, 100, 120]):
        src.append(np.full(d, n + k))
        dst.append(rng.choice(v.size, d, replace=False))
    src.append(n + 7 + np.arange(20))
    dst.append(n + 8 + np.arange(20))
    h = mg.HostGraph.from_entries(n + 28, np.concatenate(src), np.concatenate(dst))
    og = O.csr_from_arrays(*h.arrays())
    assert og.ne <= 8 * og.nv and np.max(np.diff(h.arrays()[0])) < 128
    g = mg.Graph(h)
    sources = (np.arange(count) * 3 + 5) % og.nv
    for _ in range(2):
        _check(g, og, sources, direction=direction)
    _check(g, og, [og.nv - 1, og.nv // 2], direction=direction)
    g.free()
    h.free()
