"""A level-synchronous operator defined outside the library whose labels start
at -1 (tests/plugins/hops.cu), on graphs whose small levels the built-in
operators leave to one block, on graphs with heavy rows, pushed, pulled and
switching, as one launch, as a captured loop and as a host loop: hop counts
equal to the oracle's levels."""
import ctypes as C
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))

import multigraph_gb300 as mg  # noqa: E402
from oracle import oracle as O  # noqa: E402
from plugin_build import build_plugin  # noqa: E402


def _lib():
    L = C.CDLL(build_plugin("hops"))
    L.mg_hops.argtypes = [C.c_void_p, C.c_int32, C.c_void_p, C.c_void_p, C.c_void_p]
    L.mg_hops.restype = C.c_int32
    return L


def test_operator_builds_and_exports():
    assert hasattr(_lib(), "mg_hops")


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["lattice", "path", "rmat12", "rmat18"])
def test_hops_equal_levels(kind):
    L = _lib()
    if kind == "lattice":
        h = mg.HostGraph.lattice(70, 90, 0.05, seed=2)
    elif kind == "path":
        h = mg.HostGraph.from_entries(900, np.arange(899), np.arange(1, 900))
    else:   # rows above the heavy bound; 7.6 M edges: past the one-launch form
        h = mg.HostGraph.rmat(int(kind[4:]), 16, seed=5)
    og = O.csr_from_arrays(*h.arrays())
    g = mg.Graph(h)
    for src in (0, og.nv // 3):
        want = O.bfs(og, src).astype(np.int64)
        want[want == O.IUNUSED] = -1
        for direction in (mg.DIR_AUTO, mg.DIR_PUSH, mg.DIR_PULL):
            for ex in (mg.EXEC_GRAPH, mg.EXEC_HOST):
                o = g._opts(None, dict(direction=direction, exec=ex))
                out = np.empty(g.nv, np.int32)
                assert L.mg_hops(g._h, src, C.byref(o), out.ctypes.data_as(C.c_void_p), None) == mg.MG_OK
                assert np.array_equal(out, want), (src, direction, ex)
    g.free()
    h.free()
