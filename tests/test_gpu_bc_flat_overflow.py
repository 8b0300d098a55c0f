"""Batched BC on low-degree graphs whose path counts pass 2^90 while every
level is dense (one barrier a level): the sweep ends at the same level in
every block and the run repeats with extended counts, on a fresh graph each
time.  A block that left a level early would hold the others for the barrier's
limit of about two seconds.  Scores against the long-double oracle, 1e-5
normwise (the contract of BC scores)."""
import time

import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,count", [(300, 300, 32), (130, 97, 33), (60, 1000, 5)])
def test_dense_levels_past_plain_counts(rows, cols, count):
    h = mg.HostGraph.lattice(rows, cols, 0.0, seed=3)
    og = O.csr_from_arrays(*h.arrays())
    assert og.ne <= 8 * og.nv
    src = (np.arange(count, dtype=np.int64) * 7919 + 11) % og.nv
    ref = O.bc_multi_ext(og, src)
    times = []
    for direction in (mg.DIR_PULL, mg.DIR_PULL, mg.DIR_PULL, mg.DIR_PULL, mg.DIR_AUTO, mg.DIR_PUSH):
        g = mg.Graph(h)
        t0 = time.perf_counter()
        got = g.bc_multi(src, direction=direction)[0].astype(np.float64)
        times.append(time.perf_counter() - t0)
        g.free()
        assert np.max(np.abs(got - ref)) / np.max(np.abs(ref)) < 1e-5
    h.free()
    assert max(times[1:]) < 1.5, times   # (the barrier's limit is about 2 s)
