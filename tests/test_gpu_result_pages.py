"""Results written to arrays of every kind a caller may hand in: fresh pages,
views at odd offsets, page-locked and managed memory, sizes on both sides of
1 MB (from which helper threads bring in a pageable array's pages).  Equal to
the device's results, the bytes beside the arrays untouched."""
import ctypes as C
import mmap

import numpy as np
import pytest

import multigraph_gb300 as mg
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _arrays(n):
    pad = 4096
    raw = np.full(n + 2 * pad + 1, 7, np.int32)
    yield raw, raw[pad + 1:pad + 1 + n]                       # a view inside an array
    m = mmap.mmap(-1, (n * 4 // mmap.PAGESIZE + 2) * mmap.PAGESIZE)
    whole = np.frombuffer(m, np.int32)
    yield None, whole[3:3 + n]                                # pages never touched before
    torch = pytest.importorskip("torch")
    t = torch.full((n + 2 * pad,), 7, dtype=torch.int32).pin_memory().numpy()
    yield t, t[pad:pad + n]
    rt = C.CDLL("libcudart.so.13") if _has_cudart() else None
    if rt is not None:
        p = C.c_void_p()
        assert rt.cudaMallocManaged(C.byref(p), C.c_size_t(n * 4), 1) == 0
        yield None, np.ctypeslib.as_array((C.c_int32 * n).from_address(p.value))


def _has_cudart():
    try:
        C.CDLL("libcudart.so.13")
        return True
    except OSError:
        return False


@pytest.mark.parametrize("rows,cols", [(500, 500), (512, 512), (513, 512), (2100, 1500)])
def test_result_arrays_of_every_kind(rows, cols):
    h = mg.HostGraph.lattice(rows, cols, 0.0, seed=1)
    og = O.csr_from_arrays(*h.arrays())
    g = mg.Graph(h)
    h.free()
    want = O.bfs(og, 5)
    for raw, out in _arrays(og.nv):
        g.bfs(5, out=out)
        assert np.array_equal(out, want)
        if raw is not None:
            at = (out.ctypes.data - raw.ctypes.data) // 4
            assert np.all(raw[:at] == 7) and np.all(raw[at + og.nv:] == 7)
    g.free()
