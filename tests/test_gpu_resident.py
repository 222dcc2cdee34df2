"""The resident step kernel (whole solves of small meshes in shared memory, one cooperative launch
a call) and the rules that choose it, against the tiled kernels and the oracle.

A solver without an explicit tile or block takes it where the mesh fits one tile per SM, which
launches_per_step() tells (1, the tiled kernels 2).  An explicit tile keeps the tiled kernels.  Both
form every cell's arithmetic with the same functions in the same order, so they may differ by
the fused multiply-adds the compiler picks in each kernel and no more: 1e-13 relative L-infinity in
FP64 and 1e-6 in FP32 over a few steps, the bounds the kernel families are held to elsewhere.
Against the oracle: 1e-11 after a few FP64 steps, as in the parity tests.
"""
import numpy as np
import pytest

import cfd_optimisations_b200 as H
import oracle as O

pytestmark = pytest.mark.gpu

TOL = {H.FP64: 1e-13, H.FP32: 1e-6}


def _solver(m, case, **kw):
    s = H.Solver(m, venkat_K=5.0, **kw)
    s.gather_bcs(*case[:2])
    s.initialise(case[2])
    return s


def _waves(s, seed=3):
    """A state with gradients everywhere, so that every limiter branch is taken."""
    U = s.U()
    r = np.random.default_rng(seed)
    return U * (1.0 + 0.01 * r.standard_normal(U.shape) * np.array([[1.0], [1.0], [0.0], [1.0]]))


# Sizes where it can go wrong: one tile; tiles of 32 cells; the last tile of the pair split (two
# threads a cell up to 256 cells a tile, 37,888 cells on 148 SMs) and the first beyond it; tiles with
# more cells than threads; fluxes without room of their own; the first sizes that do not fit.
SIZES = [(4, 3, True), (17, 9, True), (41, 21, True), (193, 98, True), (197, 98, True), (241, 121, True),
         (333, 178, True), (801, 401, False)]


@pytest.mark.parametrize("precision", [H.FP64, H.FP32])
@pytest.mark.parametrize("nx,ny,fits", SIZES)
def test_resident_steps_match_the_tiled_kernels(nx, ny, fits, precision):
    m = H.Mesh.wedge(nx, ny, theta_deg=10.0, seed=5, numbering=H.NUMBER_RANDOM)
    case = H.wedge_case(2.5)
    s, t = _solver(m, case, precision=precision), _solver(m, case, precision=precision, tile=128)
    assert s.launches_per_step() == (1 if fits else 2) and t.launches_per_step() == 2
    U = _waves(s)
    s.upload(U)
    t.upload(U)
    for mode, value in ((H.GLOBAL_CFL, 0.3), (H.LOCAL_CFL, 0.3), (H.FIXED_DT, 1e-5)):
        a, b = s.step(3, mode, value), t.step(3, mode, value)
        assert np.all(O.rel_linf(s.U(), t.U()) <= TOL[precision])
        assert a["dt"] == pytest.approx(b["dt"], rel=TOL[precision])
        assert a["res_l2"] == pytest.approx(b["res_l2"], rel=1e3 * TOL[precision])
        assert a["res_first"] == pytest.approx(b["res_first"], rel=1e3 * TOL[precision])
        assert a["steps"] == b["steps"]


@pytest.mark.parametrize("numbering,keep", [(H.NUMBER_RCM, True), (H.NUMBER_RANDOM, True), (H.NUMBER_RCM, False)])
@pytest.mark.parametrize("limiter", [H.LIMITER_BJ, H.LIMITER_VENKAT])
def test_resident_orders_limiters_and_boundaries_match_the_oracle(numbering, keep, limiter):
    """Input order kept (a shuffled one has halos that do not fit and takes the tiled kernels),
    every boundary type, limiter freezing."""
    m = H.Mesh.wedge(97, 49, theta_deg=8.0, seed=6, numbering=numbering)
    _, _, q = H.wedge_case(0.8)
    bcmap, qbc = np.array([H.SYMMETRY, H.WALL, H.SYMMETRY, H.SUBINLET, H.SUBOUTLET]), np.tile(q, (4, 1))
    s = _solver(m, (bcmap, qbc, q), limiter=limiter, keep_numbering=keep, freeze_limiter_after=4)
    o = O.Oracle(m.arrays())
    o.gather_bcs(bcmap, qbc)
    o.initialise(q)
    o.set_limiter(O.VENKAT if limiter == H.LIMITER_VENKAT else O.BJ, 5.0)
    o.set_freeze(4)
    s.step(8, H.GLOBAL_CFL, 0.4)
    for _ in range(8):
        o.step(O.GLOBAL_CFL, 0.4)
    assert np.all(O.rel_linf(s.U(), o.U()) <= 1e-11)


@pytest.mark.parametrize("tile", [0, 128])
@pytest.mark.parametrize("precision", [H.FP64, H.FP32])
def test_steps_in_one_call_equal_steps_one_by_one(tile, precision):
    """Also across the resident kernel's launch limit (1024 steps) and its two halves launched apart
    (profiling), and with the residual formed in the first and last steps of a call only: the
    same bits, the same first residual."""
    m = H.Mesh.wedge(61, 31, theta_deg=10.0, seed=7, numbering=H.NUMBER_RANDOM)
    case = H.wedge_case(2.5)
    a, b, c = (_solver(m, case, precision=precision, tile=tile) for _ in range(3))
    sa = a.step(1030, H.GLOBAL_CFL, 0.4)
    for _ in range(1024):
        b.step(1, H.GLOBAL_CFL, 0.4, wait=False)
    sb = b.step(6, H.GLOBAL_CFL, 0.4)
    c.profile(True, 2)
    sc = c.step(1030, H.GLOBAL_CFL, 0.4)
    p = c.profile_read()
    assert p["n_pass1"] == p["n_pass2"] == 515 and p["ms_pass1"] > 0 and p["ms_pass2"] > 0
    assert np.array_equal(a.U(), b.U()) and np.array_equal(a.U(), c.U())
    assert sa == sb == sc and sa["steps"] == 1030


def test_arena_steps_in_one_call_equal_steps_one_by_one():
    """The arena's in-between steps do their bookkeeping in pass 2 (no residual kernels): statistics
    and states of one call equal those of single steps, for instances admitted at different times."""
    from cfd_optimisations_b200.arena import Arena
    meshes = [H.Mesh.wedge(41, 21, seed=1), H.Mesh.wedge(121, 61, seed=2), H.Mesh.wedge(9, 5, seed=3)]
    bcmap, qbc, q = H.wedge_case(2.5)
    out = []
    for single in (False, True):
        a = Arena(1 << 27, precision=H.FP32)
        k = [a.admit(meshes[0], bcmap, qbc, q, 0.5)]
        for n, m in ((7, meshes[1]), (4, meshes[2]), (9, None)):
            for _ in range(n if single else 1):
                a.step(1 if single else n)
            if m is not None:
                k.append(a.admit(m, bcmap, qbc, q, 0.4))
        st = a.poll()
        out.append([(a.fetch(i), st[i]) for i in k])
    assert [x[1]["steps"] for x in out[0]] == [20, 13, 9]
    for (U, s), (V, t) in zip(*out):
        assert np.array_equal(U, V) and s == t


def test_handles_of_different_sizes_take_turns():
    """Kernels' shared-memory limits are not a handle's: a large handle steps after a smaller one
    was made, and the resident kernel of one leaves another's exchange alone."""
    case = H.wedge_case(2.5)
    meshes = [H.Mesh.wedge(nx, ny, seed=4, numbering=H.NUMBER_RANDOM) for nx, ny in ((241, 121), (17, 9))]
    for kw in ({}, dict(tile=128)):
        alone = [_solver(m, case, **kw) for m in meshes]
        for s in alone:
            s.step(6, H.GLOBAL_CFL, 0.4)
        turns = [_solver(m, case, **kw) for m in meshes]
        for _ in range(3):
            for s in turns:
                s.step(2, H.GLOBAL_CFL, 0.4, wait=False)
        for s, t in zip(alone, turns):
            assert np.array_equal(s.U(), t.U())


def test_handles_on_threads_of_their_own_step_at_the_same_time():
    """Each handle has its stream, and ctypes calls release the GIL: resident kernels that fill every
    SM, smaller ones and tiled steps at once give what they give alone (the resident
    kernel's CTAs wait for one another, so its launch is cooperative: all of them or none)."""
    import threading
    case = H.wedge_case(2.5)
    shapes = [(333, 178, {}), (333, 178, {}), (161, 81, {}), (41, 21, {}), (241, 121, dict(tile=128)), (17, 9, {})]
    meshes = [H.Mesh.wedge(nx, ny, seed=8, numbering=H.NUMBER_RANDOM) for nx, ny, _ in shapes]
    alone = []
    for m, (_, _, kw) in zip(meshes, shapes):
        s = _solver(m, case, **kw)
        st = [s.step(25, H.GLOBAL_CFL, 0.4) for _ in range(8)][-1]
        alone.append((s.U(), st))
        del s
    together = [_solver(m, case, **kw) for m, (_, _, kw) in zip(meshes, shapes)]
    got, errors = [None] * len(shapes), []

    def run(i):
        try:
            st = [together[i].step(25, H.GLOBAL_CFL, 0.4) for _ in range(8)][-1]
            got[i] = (together[i].U(), st)
        except Exception as e:                       # reported by the assertion below
            errors.append((i, e))

    threads = [threading.Thread(target=run, args=(i,)) for i in range(len(shapes))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for (U, s), (V, t) in zip(alone, got):
        assert np.array_equal(U, V) and s == t
