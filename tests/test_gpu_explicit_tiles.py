"""Tiles given explicitly, up to what shared memory holds with the plan's 16-bit face words.

(nx, ny, numbering, keep, tile, precision): a tiling of each precision whose pass 2 fits with 16-bit
face words and not with 32-bit ones, and its neighbours on either side.  States against the
per-cell kernels': 1e-13 in FP64 and 1e-6 in FP32 after a few steps, the bounds the kernel
families are held to elsewhere.
"""
import numpy as np
import pytest

import cfd_optimisations_b200 as H
import oracle as O
from poly_mesh import PolyMesh

pytestmark = pytest.mark.gpu

TOL = {H.FP64: 1e-13, H.FP32: 1e-6}
CASES = [(161, 81, H.NUMBER_RANDOM, True, 192, H.FP64), (161, 81, H.NUMBER_RANDOM, True, 160, H.FP64),
         (201, 101, H.NUMBER_RCM, True, 320, H.FP64), (201, 101, H.NUMBER_RCM, True, 288, H.FP64),
         (1025, 513, H.NUMBER_RCM, True, 448, H.FP32)]


@pytest.mark.parametrize("nx,ny,numbering,keep,tile,precision", CASES)
@pytest.mark.parametrize("mode", [H.GLOBAL_CFL, H.LOCAL_CFL])
def test_explicit_tiles_match_the_per_cell_kernels(nx, ny, numbering, keep, tile, precision, mode):
    m = H.Mesh.wedge(nx, ny, theta_deg=10.0, seed=3, numbering=numbering)
    bcmap, qbc, q = H.wedge_case(2.5)
    got = []
    for kw in (dict(tile=tile, keep_numbering=keep), dict(kernel=H.KERNEL_CELL, keep_numbering=keep)):
        s = H.Solver(m, precision=precision, **kw)
        s.gather_bcs(bcmap, qbc)
        s.initialise(q)
        st = s.step(4, mode, 0.4)
        got.append((s.U(), st))
        del s
    (U, a), (V, b) = got
    assert np.all(O.rel_linf(U, V) <= TOL[precision])
    assert a["dt"] == pytest.approx(b["dt"], rel=TOL[precision])
    assert a["res_l2"] == pytest.approx(b["res_l2"], rel=1e3 * TOL[precision])


# Cells of three to eight faces, FP64: 16-bit words in pass 2 (352) and in pass 1 (480), and neither (320).
@pytest.mark.parametrize("nx,ny,kw", [(90, 45, dict(tile=352)), (90, 24, dict(tile=480, tile2=128)), (90, 45, dict(tile=320))])
@pytest.mark.parametrize("limiter", [H.LIMITER_BJ, H.LIMITER_VENKAT])
def test_wide_cells(nx, ny, kw, limiter):
    m, q = PolyMesh(nx, ny), (1.4, 2.2, 0.35, 1.0)
    r = np.random.default_rng(3)
    U, got = None, []
    for k in (kw, dict(kernel=H.KERNEL_CELL)):
        s = H.Solver(m, limiter=limiter, venkat_K=5.0, **k)
        s.gather_bcs([H.SYMMETRY, H.SYMMETRY, H.SUPOUTLET, H.WALL, H.SUPINLET], [q] * 4)
        s.initialise(q)
        if U is None:
            U = s.U() * (1.0 + 0.01 * r.standard_normal((4, m.Nc)) * np.array([[1.0], [1.0], [0.0], [1.0]]))
        s.upload(U)
        st = s.step(4, H.GLOBAL_CFL, 0.3)
        got.append((s.U(), st["dt"]))
    assert np.all(O.rel_linf(got[0][0], got[1][0]) <= TOL[H.FP64])
    assert got[0][1] == pytest.approx(got[1][1], rel=TOL[H.FP64])
