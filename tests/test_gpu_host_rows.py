"""Read-backs and uploads into four host arrays that lie end to end, page-locked one by one.

The four rows of a C-contiguous array are moved in one copy where their memory is pageable; rows
registered on their own are separate registrations, which one copy may not cross."""
import mmap

import numpy as np
import pytest

import cfd_optimisations_b200 as H
from cfd_optimisations_b200.arena import Arena

pytestmark = pytest.mark.gpu

PAGE = mmap.PAGESIZE


@pytest.mark.parametrize("rows", [(0, 1, 2, 3), (1,), (2, 3), (3,)])
def test_rows_pinned_one_by_one(rows):
    m = H.Mesh.wedge(27, 19, seed=2)
    assert 8 * m.Nc % PAGE == 0                      # a row ends on a page: neighbours share none
    bcmap, qbc, q = H.wedge_case(2.5)
    s = H.Solver(m)
    s.gather_bcs(bcmap, qbc)
    s.initialise(q)
    s.step(5, H.GLOBAL_CFL, 0.4)
    want, prims = s.U(), s.Q()
    buf = mmap.mmap(-1, 4 * 8 * m.Nc)                # page-aligned
    a = np.frombuffer(buf, dtype=np.float64).reshape(4, m.Nc)
    for r in rows:
        H.pin(a[r])
    try:
        for kw, w in (({}, want), (dict(prims=True), prims)):
            a[:] = 0.0
            s.download(out=a, **kw)
            assert np.array_equal(a, w)
        a[:] = want * 1.25
        s.upload(a)
        assert np.array_equal(s.U(), want * 1.25)
    finally:
        for r in rows:
            H.unpin(a[r])


def test_arena_fetch_into_pinned_rows():
    import ctypes as ct
    from cfd_optimisations_b200 import native as N
    m = H.Mesh.wedge(27, 19, seed=2)
    bcmap, qbc, q = H.wedge_case(2.5)
    ar = Arena(1 << 26, precision=H.FP64)
    k = ar.admit(m, bcmap, qbc, q, 0.4)
    ar.step(5)
    want = ar.fetch(k)
    buf = mmap.mmap(-1, 4 * 8 * m.Nc)
    a = np.frombuffer(buf, dtype=np.float64).reshape(4, m.Nc)
    for r in a:
        H.pin(r)
    try:
        ptrs = (N._dp * 4)(*[r.ctypes.data_as(N._dp) for r in a])
        N.check(N.lib().hcfd_arena_fetch(ar._h, k, 0, ptrs))
        assert np.array_equal(a, want)
    finally:
        for r in a:
            H.unpin(r)
