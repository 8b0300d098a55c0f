"""A seed's personalised ranks do not depend on how many seeds share its pass:
rows of any length are summed in the same order whatever the pass's width.
Rows of 1 to 40 chunks of 256 edges, bit for bit over passes of 1, 5, 9, 17
and 32 copies of a seed; 2e-7 absolute from the FP64 oracle after the same
sweeps."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _graph():
    rng = np.random.default_rng(4)
    n = 12_000
    src, dst = [rng.integers(0, n, 4 * n)], [rng.integers(0, n, 4 * n)]
    for k, d in enumerate([255, 256, 257, 512, 513, 1025, 2047, 2048, 2049, 2305, 4096, 8192, 8193, 10_200]):
        src.append(np.full(d, n + k))
        dst.append(rng.choice(n, d, replace=False))
    return mg.HostGraph.from_entries(n + 14, np.concatenate(src), np.concatenate(dst))


def test_ranks_do_not_depend_on_the_pass_width():
    h = _graph()
    og = O.csr_from_arrays(*h.arrays())
    g = mg.Graph(h)
    for seed in (0, og.nv - 1, og.nv // 2):
        one, info = g.ppr_batch([seed], tol=1e-6)
        ref = O.ppr_f64(og, seed, 0.85, 1e-30, info.iterations)[0]
        assert np.max(np.abs(one[0] - ref)) < 2e-7
        for count in (5, 9, 17, 32):
            many, i2 = g.ppr_batch([seed] * count, tol=1e-6)
            assert i2.iterations == info.iterations
            for row in many:
                assert np.array_equal(row, one[0]), count
    g.free()
    h.free()
