"""Steps profiled half by half leave nothing behind that a later whole step takes for its own.

The resident kernel's tiles exchange words that carry a step's stamp, and its profiled halves pass
the limited gradients of all cells through the same memory.  The state here has a momentum gradient
so small (a denormal) that its upper words are the stamp of a coming step: with the old words
still there, that step would read them as its neighbours'.  A profiled step and a plain one
equal two plain ones bit for bit, as for any other state (test_gpu_resident.py).
"""
import numpy as np
import pytest

import cfd_optimisations_b200 as H

pytestmark = pytest.mark.gpu


def _solver(m):
    s = H.Solver(m)
    bcmap, qbc, q = H.wedge_case(2.5)
    s.gather_bcs(bcmap, qbc)
    s.initialise(q)
    return s


@pytest.mark.parametrize("stamp", [3, 4, 5])
def test_a_plain_step_after_a_profiled_one(stamp):
    m = H.Mesh.wedge(161, 81, theta_deg=2.0, jitter=0.0, seed=1, numbering=H.NUMBER_RCM)
    a = m.arrays()
    xy = a["nodes"].reshape(-1, 2)
    off = a["cn_off"]
    centre = np.add.reduceat(xy[a["cn_con"]], off[:-1], axis=0) / np.diff(off)[:, None]
    # the smallest double whose upper 32 bits are `stamp`, and half as much again of the range above
    slope = (stamp + 0.5) * np.frombuffer(np.int64(1 << 32).tobytes(), dtype=np.float64)[0]
    U = np.empty((4, m.Nc))
    U[0], U[3] = 1.4, 2.5
    U[1] = U[2] = slope * (centre[:, 0] + centre[:, 1])
    plain, profiled = _solver(m), _solver(m)
    assert plain.launches_per_step() == 1
    for s in (plain, profiled):
        s.upload(U)
    profiled.profile(True)
    profiled.step(1, H.FIXED_DT, 1e-6)
    profiled.profile(False)
    plain.step(1, H.FIXED_DT, 1e-6)
    assert np.array_equal(plain.U(), profiled.U())
    for s in (plain, profiled):
        s.step(3, H.FIXED_DT, 1e-6)
    assert np.array_equal(plain.U(), profiled.U())
