"""The mesh of many-sided cells is what its tests say it is, and its tile plans hold (no GPU needed)."""
import numpy as np
import pytest

import cfd_optimisations_b200 as H
import oracle as O
from poly_mesh import PolyMesh


def test_cells_have_three_to_eight_faces_and_keep_a_uniform_flow():
    m = PolyMesh(40, 20)
    a = m.arrays()
    real = a["Nc"] - (a["Nf"] - a["coloff"][1])
    faces = np.bincount(a["fc_con"], minlength=a["Nc"])[:real]
    assert set(faces) == {3, 4, 5, 6, 7, 8}
    o = O.Oracle(a)
    q = [1.4, 2.5, 0.3, 1.0]
    o.gather_bcs([O.SYMMETRY] + [O.SUPINLET] * 4, [q] * 4)
    o.initialise(q)
    U0 = o.U()
    for _ in range(5):
        o.step(O.GLOBAL_CFL, 0.4)
    assert np.all(O.rel_linf(o.U(), U0) <= 1e-13)


@pytest.mark.parametrize("tile", [32, 40, 128, 256])
def test_plans_of_eight_slots(tile):
    assert H.plan_check(PolyMesh(60, 30), tile=tile)["slots"] == 8
