"""One-launch PageRank is no further from the FP64 recurrence after the same
sweeps than the named layouts on the same graphs (geometric mean of the
relative root mean square errors over graphs with rows of every kind)."""
import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_error_against_64_bits():
    logs = {None: [], mg.PR_LAYOUT_GATHER: [], mg.PR_LAYOUT_SEGMENTED: []}
    graphs = [mg.HostGraph.rmat(k, ef, seed=s) for k, ef, s in
              [(9, 7, 1), (10, 16, 2), (11, 24, 3), (12, 20, 4), (13, 8, 5), (14, 16, 6), (15, 18, 7), (16, 16, 8)]]
    for h in graphs:
        og = O.csr_from_arrays(*h.arrays())
        g = mg.Graph(h)
        for layout, out in logs.items():
            kw = {} if layout is None else dict(pr_layout=layout)
            x, info = g.pagerank(mg.PR_TOPOLOGY, tol=1e-6, **kw)
            ref, _ = O.pr_norm_f64(og, float(np.float32(0.85)), 1e-30, info.iterations)
            out.append(np.log(np.sqrt(np.mean((x - ref) ** 2) / np.mean(ref ** 2))))
        g.free()
        h.free()
    err = {k: float(np.exp(np.mean(v))) for k, v in logs.items()}
    assert err[None] <= min(err[mg.PR_LAYOUT_GATHER], err[mg.PR_LAYOUT_SEGMENTED]), err
