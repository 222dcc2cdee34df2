"""Venkatakrishnan's limiter for every sign of its constant.

With K > 0 the face with the largest increment on each side decides, whatever the number of faces;
with K < 0 (e2 = (K h)^3 < 0) it does not, and every face is looked at.  |K| is large enough here
that e2 outweighs the other terms (numerator and denominator keep their sign) and the limiter stays well
conditioned.  One step from a state with gradients everywhere against the oracle: 1e-12, the
one-step tolerance of the parity tests; FP32 against the per-cell FP32 kernels, 1e-6.
"""
import numpy as np
import pytest

import cfd_optimisations_b200 as H
import oracle as O
from cfd_optimisations_b200.arena import Arena
from poly_mesh import PolyMesh

pytestmark = pytest.mark.gpu

KS = [-500.0, -0.0, 0.0, 5.0]
KERNELS = [dict(), dict(tile=128), dict(tile=256, tile2=128), dict(kernel=H.KERNEL_CELL)]


def _state(U):
    r = np.random.default_rng(3)
    return U * (1.0 + 0.01 * r.standard_normal(U.shape) * np.array([[1.0], [1.0], [0.0], [1.0]]))


def _case():
    m = H.Mesh.wedge(81, 41, theta_deg=10.0, seed=5, numbering=H.NUMBER_RANDOM)
    return m, H.wedge_case(2.5)


def _solver(m, case, **kw):
    s = H.Solver(m, limiter=H.LIMITER_VENKAT, **kw)
    s.gather_bcs(*case[:2])
    s.initialise(case[2])
    return s


@pytest.mark.parametrize("K", KS)
@pytest.mark.parametrize("kw", KERNELS)
def test_one_step_matches_the_oracle(kw, K):
    m, case = _case()
    s = _solver(m, case, venkat_K=K, **kw)
    U = _state(s.U())
    o = O.Oracle(m.arrays())
    o.gather_bcs(*case[:2])
    o.initialise(case[2])
    o.set_limiter(O.VENKAT, K)
    s.upload(U)
    o.set_U(U)
    s.step(1, H.GLOBAL_CFL, 0.4)
    o.step(O.GLOBAL_CFL, 0.4)
    assert np.all(O.rel_linf(s.U(), o.U()) <= 1e-12)


@pytest.mark.parametrize("K", [KS[0], KS[-1]])
@pytest.mark.parametrize("kw", KERNELS[1:])
def test_wide_cells_match_the_oracle(kw, K):
    q = (1.4, 2.2, 0.35, 1.0)
    m, case = PolyMesh(60, 30), ([H.SYMMETRY, H.SYMMETRY, H.SUPOUTLET, H.WALL, H.SUPINLET], [q] * 4, q)
    s = _solver(m, case, venkat_K=K, **kw)
    U = _state(s.U())
    o = O.Oracle(m.arrays())
    o.gather_bcs(*case[:2])
    o.initialise(q)
    o.set_limiter(O.VENKAT, K)
    s.upload(U)
    o.set_U(U)
    s.step(1, H.GLOBAL_CFL, 0.4)
    o.step(O.GLOBAL_CFL, 0.4)
    assert np.all(O.rel_linf(s.U(), o.U()) <= 1e-12)


@pytest.mark.parametrize("kw", KERNELS[1:3])
def test_fp32_kernels_agree(kw):
    m, case = _case()
    a, b = (_solver(m, case, venkat_K=-500.0, precision=H.FP32, **k) for k in (kw, dict(kernel=H.KERNEL_CELL)))
    U = _state(a.U())
    for s in (a, b):
        s.upload(U)
        s.step(3, H.LOCAL_CFL, 0.3)
    assert np.all(O.rel_linf(a.U(), b.U()) <= 1e-6)


@pytest.mark.parametrize("precision,tol", [(H.FP64, 1e-13), (H.FP32, 1e-6)])
def test_arena_agrees_with_the_tiled_solver(precision, tol):
    m, case = _case()
    s = _solver(m, case, venkat_K=-500.0, precision=precision, tile=128)
    ar = Arena(1 << 27, precision=precision, limiter=H.LIMITER_VENKAT, venkat_K=-500.0)
    k = ar.admit(m, *case, 0.4)
    ar.step(10)
    s.step(10, H.GLOBAL_CFL, 0.4)
    assert np.all(O.rel_linf(ar.fetch(k), s.U()) <= tol)


def test_noalloc_step_with_a_negative_constant():
    from test_zz_no_alloc import _noalloc_case
    m, case = _case()
    assert _noalloc_case(m, *case, H.LIMITER_VENKAT, -500.0, H.GLOBAL_CFL, 0.4) == 3
