"""Bounded waits that run out, on every step kernel: the call reports HCFD_ETIMEOUT, no copy outlives
its CTA, and the re-initialised handle steps bit-identically to a fresh one.

test_gpu_waits.py holds the general statement and its reasons; here each kernel is named by its launch
shape and launches_per_step().  No GPU fault is made: every address stays valid.
"""
import numpy as np
import pytest

import cfd_optimisations_b200 as H
from cfd_optimisations_b200 import native as N

pytestmark = pytest.mark.gpu

# (nx, ny, Solver keywords, launches per step): the tiled kernels on one plan and on two, and the
# resident kernel with two threads a cell, with one, and with fluxes over the refetched r vectors
TILED = [(201, 101, dict(tile=128)), (201, 101, dict(tile=256, tile2=128)), (401, 201, dict(tile=128))]
RESIDENT = {H.FP64: [(81, 41, {}), (333, 178, {}), (361, 181, {})], H.FP32: [(81, 41, {}), (333, 178, {}), (501, 251, {})]}
CASES = [(p, 2, *c) for p in (H.FP64, H.FP32) for c in TILED] + [(p, 1, *c) for p, l in RESIDENT.items() for c in l]


def _solver(m, precision, kw):
    s = H.Solver(m, precision=precision, limiter=H.LIMITER_VENKAT, venkat_K=5.0, **kw)
    bcmap, qbc, q = H.wedge_case(2.5)
    s.gather_bcs(bcmap, qbc)
    s.initialise(q)
    return s


def _recovers(s, m, precision, kw):
    N.check(N.lib().hcfd_gpu_test_waits(s._h, 0, -1))
    s.initialise(H.wedge_case(2.5)[2])
    st = s.step(6, H.GLOBAL_CFL, 0.5)
    fresh = _solver(m, precision, kw)
    st_f = fresh.step(6, H.GLOBAL_CFL, 0.5)
    assert np.array_equal(s.U(), fresh.U()) and st == st_f


@pytest.mark.parametrize("precision,launches,nx,ny,kw", CASES)
def test_a_poll_limit_of_one(precision, launches, nx, ny, kw):
    """Compute warps may give up before their first tile is armed in full, whose tables are copied while
    the kernel before still runs.  Whether a wait runs out depends on the copies' speed; what
    follows does not."""
    m = H.Mesh.wedge(nx, ny, seed=9, numbering=H.NUMBER_RCM)
    s = _solver(m, precision, kw)
    assert s.launches_per_step() == launches
    N.check(N.lib().hcfd_gpu_test_waits(s._h, 1, -1))
    for steps in (1, 2, 5):
        try:
            s.step(steps, H.GLOBAL_CFL, 0.5)
        except H.HcfdError as e:
            assert e.code == N.ETIMEOUT
    _recovers(s, m, precision, kw)


@pytest.mark.parametrize("skip", [0, 1])
@pytest.mark.parametrize("mode,value", [(H.GLOBAL_CFL, 0.5), (H.FIXED_DT, 1e-5)])
@pytest.mark.parametrize("precision,launches,nx,ny,kw", CASES)
def test_a_tile_that_never_arrives(precision, launches, nx, ny, kw, mode, value, skip):
    """In the resident kernel a fixed step holds no tile back but a neighbour, so tiles far from the
    missing one give up some steps later, with their r vectors' copies of the next step in flight
    where fluxes take those vectors' room."""
    m = H.Mesh.wedge(nx, ny, seed=9, numbering=H.NUMBER_RCM)
    s = _solver(m, precision, kw)
    assert s.launches_per_step() == launches
    s.step(2, H.GLOBAL_CFL, 0.5)
    N.check(N.lib().hcfd_gpu_test_waits(s._h, 1 << 14, skip))
    with pytest.raises(H.HcfdError) as e:
        s.step(40 if launches == 1 else 2, mode, value)
    assert e.value.code == N.ETIMEOUT
    with pytest.raises(H.HcfdError):
        s.sync()
    _recovers(s, m, precision, kw)
