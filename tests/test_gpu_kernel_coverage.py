"""Every step kernel on the meshes and options it accepts, the kernel named in each case by its launch shape
and launches_per_step(): the resident kernel (no explicit tile), the tiled kernels on one plan
(8-value face records) and on two (7-value records in pass 2).

FP64 against the oracle: 1e-11 after eight steps, as in the parity tests; FP32 against the per-cell FP32
kernels: 1e-6 after a few steps, the bound the kernel families are held to elsewhere.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
if __name__ == "__main__":
    sys.path[:0] = [os.path.dirname(HERE), os.path.join(os.path.dirname(HERE), "oracle"), HERE]

import cfd_optimisations_b200 as H  # noqa: E402
import oracle as O  # noqa: E402
from poly_mesh import PolyMesh  # noqa: E402

pytestmark = pytest.mark.gpu

KERNELS = {"resident": ({}, 1), "one_plan": (dict(tile=128), 2), "two_plans": (dict(tile=256, tile2=128), 2),
           "small_tiles": (dict(tile=64, tile2=32), 2)}
TOL = {H.FP64: 1e-13, H.FP32: 1e-6}


def _mesh(kind, tmp):
    """The mesh, boundary map, boundary states and initial state of a kind: three faces a cell with every
    subsonic boundary type and a wall, four (quadrangles and triangles), and three to eight."""
    if kind == "triangles":
        m = H.Mesh.wedge(97, 49, theta_deg=8.0, seed=6, numbering=H.NUMBER_RANDOM)
        _, _, q = H.wedge_case(0.8)
        return m, [H.SYMMETRY, H.WALL, H.SYMMETRY, H.SUBINLET, H.SUBOUTLET], np.tile(q, (4, 1)), q
    q = (1.4, 2.2, 0.35, 1.0)
    bcmap = [H.SYMMETRY, H.SYMMETRY, H.SUPOUTLET, H.WALL, H.SUPINLET]
    if kind == "mixed":
        from test_meshio import write_msh
        from cfd_optimisations_b200 import meshio
        write_msh(os.path.join(tmp, "r.msh"), nx=61, ny=31)
        meshio.import_msh(os.path.join(tmp, "r.msh"), os.path.join(tmp, "r.hmsh"))
        return H.Mesh(os.path.join(tmp, "r.hmsh")), bcmap, [q] * 4, q
    return PolyMesh(90, 45), bcmap, [q] * 4, q


def _solver(case, precision=H.FP64, launches=None, **kw):
    m, bcmap, qbc, q = case
    s = H.Solver(m, precision=precision, venkat_K=5.0, **kw)
    assert launches is None or s.launches_per_step() == launches
    s.gather_bcs(bcmap, qbc)
    s.initialise(q)
    return s


def _waves(U):
    r = np.random.default_rng(3)
    return U * (1.0 + 0.01 * r.standard_normal(U.shape) * np.array([[1.0], [1.0], [0.0], [1.0]]))


@pytest.mark.parametrize("freeze", [0, 4])
@pytest.mark.parametrize("limiter", [H.LIMITER_BJ, H.LIMITER_VENKAT])
@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("kind", ["triangles", "mixed", "poly"])
def test_kernels_match_the_oracle(kind, kernel, limiter, freeze, tmp_path):
    case = _mesh(kind, str(tmp_path))
    kw, launches = KERNELS[kernel]
    s = _solver(case, launches=launches, limiter=limiter, freeze_limiter_after=freeze, **kw)
    U = _waves(s.U())
    for mode, value in ((H.GLOBAL_CFL, 0.3), (H.LOCAL_CFL, 0.3), (H.FIXED_DT, 1e-5)):
        o = O.Oracle(case[0].arrays())
        o.gather_bcs(case[1], case[2])
        o.initialise(case[3])
        o.set_limiter(O.VENKAT if limiter == H.LIMITER_VENKAT else O.BJ, 5.0)
        o.set_freeze(freeze)
        s.initialise(case[3])
        s.upload(U)
        o.set_U(U)
        st = s.step(8, mode, value)
        for _ in range(8):
            dt, res = o.step(mode, value)
        assert np.all(O.rel_linf(s.U(), o.U()) <= 1e-11), (mode, O.rel_linf(s.U(), o.U()))
        assert st["dt"] == pytest.approx(dt, rel=1e-11) and st["res_l2"] == pytest.approx(res, rel=1e-8)


@pytest.mark.parametrize("limiter", [H.LIMITER_BJ, H.LIMITER_VENKAT])
@pytest.mark.parametrize("kernel", KERNELS)
@pytest.mark.parametrize("kind", ["triangles", "mixed", "poly"])
def test_fp32_kernels_match_the_per_cell_ones(kind, kernel, limiter, tmp_path):
    case = _mesh(kind, str(tmp_path))
    kw, launches = KERNELS[kernel]
    s = _solver(case, H.FP32, launches, limiter=limiter, freeze_limiter_after=5, **kw)
    c = _solver(case, H.FP32, 2, limiter=limiter, freeze_limiter_after=5, kernel=H.KERNEL_CELL)
    U = _waves(s.U())
    s.upload(U)
    c.upload(U)
    for mode, value in ((H.GLOBAL_CFL, 0.3), (H.LOCAL_CFL, 0.3), (H.FIXED_DT, 1e-5)):
        a, b = s.step(3, mode, value), c.step(3, mode, value)
        assert np.all(O.rel_linf(s.U(), c.U()) <= 1e-6), (mode, O.rel_linf(s.U(), c.U()))
        assert a["dt"] == pytest.approx(b["dt"], rel=1e-6)


# The largest sizes of the resident kernel on 148 SMs (fluxes over the r vectors at the first and third),
# and the first beyond them.
@pytest.mark.parametrize("nx,ny,precision,launches", [(361, 181, H.FP64, 1), (369, 185, H.FP64, 2), (457, 229, H.FP32, 1),
                                                      (501, 251, H.FP32, 1), (513, 257, H.FP32, 2)])
def test_resident_kernel_at_its_capacity(nx, ny, precision, launches):
    m = H.Mesh.wedge(nx, ny, theta_deg=10.0, seed=5, numbering=H.NUMBER_RANDOM)
    case = (m, *H.wedge_case(2.5))
    s = _solver(case, precision, launches)
    t = _solver(case, precision, 2, tile=128)
    U = _waves(s.U())
    s.upload(U)
    t.upload(U)
    for mode, value in ((H.GLOBAL_CFL, 0.3), (H.LOCAL_CFL, 0.3), (H.FIXED_DT, 1e-5)):
        a, b = s.step(3, mode, value), t.step(3, mode, value)
        assert np.all(O.rel_linf(s.U(), t.U()) <= TOL[precision])
        assert a["dt"] == pytest.approx(b["dt"], rel=TOL[precision])


def test_checked_build_on_every_kernel(tmp_path):
    """The checked build finds no index out of range on these meshes and changes no state beyond what
    the kernel families may differ by."""
    runs = {}
    for which in ("default", "checked"):
        out = str(tmp_path / f"{which}.npz")
        r = subprocess.run([sys.executable, os.path.abspath(__file__), out], env=dict(os.environ, HCFD_LIB=which),
                           capture_output=True, text=True, timeout=900)
        assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]
        runs[which] = np.load(out)
    d, c = runs["default"], runs["checked"]
    assert sorted(d.files) == sorted(c.files) and len(d.files) == 26
    for k in d.files:
        assert np.all(O.rel_linf(c[k], d[k]) <= TOL[H.FP32 if "fp32" in k else H.FP64]), k


def _checked_runs(out):
    import tempfile
    res = {}
    with tempfile.TemporaryDirectory() as tmp:
        for kind in ("triangles", "mixed", "poly"):
            case = _mesh(kind, tmp)
            for kernel, (kw, launches) in KERNELS.items():
                for name, precision in (("fp64", H.FP64), ("fp32", H.FP32)):
                    s = _solver(case, precision, launches, freeze_limiter_after=4, **kw)
                    s.upload(_waves(s.U()))
                    s.step(3, H.GLOBAL_CFL, 0.3)
                    s.step(3, H.LOCAL_CFL, 0.3)
                    res[f"{kind}_{kernel}_{name}"] = s.U()
    # 16-bit face words, on one plan and as the default's fallback
    case = (H.Mesh.wedge(161, 81, theta_deg=10.0, seed=3, numbering=H.NUMBER_RANDOM), *H.wedge_case(2.5))
    for name, kw in (("short_words", dict(tile=192)), ("short_words_two_plans", dict(tile=64, tile2=192))):
        s = _solver(case, H.FP64, 2, keep_numbering=True, **kw)
        s.step(6, H.GLOBAL_CFL, 0.3)
        res[name + "_fp64"] = s.U()
    np.savez(out, **res)


if __name__ == "__main__":
    _checked_runs(sys.argv[1])
