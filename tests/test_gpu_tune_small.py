"""MG_PR_LAYOUT_AUTO on a graph small enough for PageRank in one launch: the
default is that form; mg_autotune times it against the tuned layouts, records
the outcome and AUTO follows the record; lines of a cache file from before the
record leave the default.  The three routes are told apart by their bits."""
import os
import tempfile

import numpy as np
import pytest

import multigraph_gb300 as mg

pytestmark = pytest.mark.gpu


def _run(g, layout=None):
    kw = {} if layout is None else dict(pr_layout=layout)
    return g.pagerank(mg.PR_TOPOLOGY, tol=1e-6, **kw)[0]


def test_auto_follows_the_record():
    h = mg.HostGraph.rmat(15, 16, seed=7)
    g = mg.Graph(h)
    default = _run(g)
    cache = os.path.join(tempfile.mkdtemp(), "tune.txt")
    g.autotune(mg.ALGO_PR, 0, cache)
    words = open(cache).read().split()
    assert len(words) == 8 and words[6] in "01" and words[7] in "01"
    named = {1: _run(g, mg.PR_LAYOUT_SEGMENTED), 0: _run(g, mg.PR_LAYOUT_GATHER)}
    for x in named.values():
        assert not np.array_equal(x, default)
    assert not np.array_equal(named[0], named[1])
    assert np.array_equal(_run(g), default if words[7] == "1" else named[int(words[6])])
    g.free()
    for layout in ("0", "1"):
        for one in ("0", "1", None):
            with open(cache, "w") as f:
                f.write(" ".join(words[:6] + [layout] + ([one] if one else [])) + "\n")
            g = mg.Graph(h)
            g.autotune(mg.ALGO_PR, 0, cache)
            want = named[int(layout)] if one == "0" else default
            assert np.array_equal(_run(g), want), (layout, one)
            g.free()
    # a graph laid out anew has not been timed: the default again
    with open(cache, "w") as f:
        f.write(" ".join(words[:6] + ["1", "0"]) + "\n")
    g = mg.Graph(h)
    g.autotune(mg.ALGO_PR, 0, cache)
    row, col, wt = h.arrays()
    perm = np.random.default_rng(1).permutation(h.nv)
    other = mg.HostGraph.from_entries(h.nv, perm[np.repeat(np.arange(h.nv), np.diff(row))], perm[col], wt,
                                      flags=mg.LOAD_NSYM)
    assert (other.nv, other.ne) == (h.nv, h.ne)
    fresh = mg.Graph(other)
    g.reload(other)
    assert np.array_equal(_run(g), _run(fresh))
    for x in (g, fresh):
        x.free()
    h.free()
    other.free()
