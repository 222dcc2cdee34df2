"""A step under a CFL number takes the minimum of its own state, whatever steps came before it:
a fixed step in between, or a state with a larger step uploaded.

The sequences are of single steps, an odd number of them between two CFL steps, so that the
second uses the same minimum slot as the first.  dt against the oracle's: 1e-13 (a maximum
of the cells' rates and one reciprocal, as in the parity tests), FP32 1e-5.
"""
import numpy as np
import pytest

import cfd_optimisations_b200 as H
import oracle as O

pytestmark = pytest.mark.gpu

KERNELS = [(dict(), 1), (dict(tile=128), 2), (dict(tile=256, tile2=128), 2), (dict(kernel=H.KERNEL_CELL), 2)]


@pytest.mark.parametrize("precision,tol", [(H.FP64, 1e-13), (H.FP32, 1e-5)])
@pytest.mark.parametrize("between", [H.FIXED_DT, H.LOCAL_CFL])
@pytest.mark.parametrize("kw,launches", KERNELS)
def test_cfl_step_after_other_steps(kw, launches, between, precision, tol):
    m = H.Mesh.wedge(61, 31, theta_deg=10.0, seed=12, numbering=H.NUMBER_RANDOM)
    bcmap, qbc, q = H.wedge_case(2.5)
    s = H.Solver(m, precision=precision, **kw)
    assert s.launches_per_step() == launches
    s.gather_bcs(bcmap, qbc)
    s.initialise(q)
    o = O.Oracle(m.arrays())
    o.gather_bcs(bcmap, qbc)
    o.initialise(q)
    first = s.step(1, H.GLOBAL_CFL, 0.4)["dt"]
    assert first == pytest.approx(o.step(O.GLOBAL_CFL, 0.4)[0], rel=tol)
    s.step(1, between, 1e-6 if between == H.FIXED_DT else 0.1)
    # a slower gas: its step is longer than the first one's
    slow = s.U()
    slow[1:3] *= 0.1
    slow[3] = 1.0 / 0.4 + 0.5 * (slow[1] ** 2 + slow[2] ** 2) / slow[0]
    s.upload(slow)
    o.set_U(s.U())
    want = o.step(O.GLOBAL_CFL, 0.4)[0]
    assert want > 1.2 * first
    assert s.step(1, H.GLOBAL_CFL, 0.4)["dt"] == pytest.approx(want, rel=tol)
    # two fixed steps and one: the other slot
    s.step(2, H.FIXED_DT, 1e-6)
    s.upload(slow * 1.0)
    assert s.step(1, H.GLOBAL_CFL, 0.4)["dt"] == pytest.approx(want, rel=tol)
    assert np.all(np.isfinite(s.U()))
