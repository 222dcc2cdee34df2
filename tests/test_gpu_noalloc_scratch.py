"""The allocation-free step owes nothing to the calls before it: each call starts its scratch over.

Every case runs in a process of its own, since the scratch belongs to a context and what is looked
at is the context's first calls.  The reference of each step is the per-cell solver in the
caller's numbering, whose kernels do the same arithmetic (ONE_STEP of test_zz_no_alloc.py).

    python tests/test_gpu_noalloc_scratch.py CASE
"""
import ctypes as ct
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ONE_STEP = 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("case", ["after_refused", "captured"])
def test_noalloc_scratch(case):
    r = subprocess.run([sys.executable, os.path.abspath(__file__), case], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-4000:]


class _Case:
    """The small wedge of checked_cases.py in the caller's buffers, and two CFL steps of the solver."""

    def __init__(self):
        import torch
        from checked_cases import _noalloc_setup
        import cfd_optimisations_b200 as H
        import oracle as O
        self.torch, self.H, self.O = torch, H, O
        self.m, self.bufs, self.Nc, _, _ = _noalloc_setup()
        self.start = self.bufs["d_U"][0].clone()
        mesh = H.Mesh.wedge(81, 41, theta_deg=15.0, seed=17, numbering=H.NUMBER_RANDOM)
        s = H.Solver(mesh, kernel=H.KERNEL_CELL, keep_numbering=True, limiter=H.LIMITER_VENKAT, venkat_K=5.0)
        bcmap, qbc, q = H.wedge_case(2.5)
        s.gather_bcs(bcmap, qbc)
        s.initialise(q)
        self.ref = []
        for _ in range(2):
            st = s.step(1, H.GLOBAL_CFL, 0.5)
            self.ref.append((s.U(), st["dt"]))

    def call(self, src, dst, mode, value, stream=None, stats=True):
        from cfd_optimisations_b200 import native as N
        dt, res = ct.c_double(), ct.c_double()
        rc = N.lib().hcfd_step_noalloc(ct.byref(self.m), src.data_ptr(), dst.data_ptr(), mode, value, stream,
                                       ct.byref(dt) if stats else None, ct.byref(res) if stats else None)
        return rc, dt.value

    def check(self, buf, i):
        from test_zz_no_alloc import _unplanes
        self.torch.cuda.synchronize()
        err = self.O.rel_linf(_unplanes(buf.cpu().numpy(), self.Nc), self.ref[i][0])
        assert np.all(err <= ONE_STEP), err

    def two_steps(self):
        a, b = self.bufs["d_U"]
        a.copy_(self.start)
        self.torch.cuda.synchronize()
        for i, (src, dst) in enumerate(((a, b), (b, a))):
            rc, dt = self.call(src, dst, self.H.GLOBAL_CFL, 0.5)
            assert rc == 0 and abs(dt - self.ref[i][1]) <= 1e-13 * self.ref[i][1], (rc, dt, self.ref[i][1])
            self.check(dst, i)

    def refused_call(self):
        """A first call that is refused for its boundary type."""
        from cfd_optimisations_b200 import native as N
        types = self.bufs["bc_type"]
        keep = int(types[0])
        types[0] = 99
        rc, _ = self.call(*self.bufs["d_U"], self.H.GLOBAL_CFL, 0.5)
        types[0] = keep
        assert rc == N.EINVAL


def _after_refused():
    c = _Case()
    c.refused_call()
    c.two_steps()


def _captured():
    """Two steps captured on the caller's stream after a first, direct one (as the header asks), a
    direct step before the graph has run, then replays with direct steps in between."""
    c = _Case()
    torch = c.torch
    a, b = c.bufs["d_U"]
    assert c.call(a, b, c.H.FIXED_DT, 1e-6)[0] == 0
    s = torch.cuda.Stream()
    x, y = c.start.clone(), torch.zeros_like(c.start)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        for src, dst in ((x, y), (y, x)):
            rc, _ = c.call(src, dst, c.H.GLOBAL_CFL, 0.5, s.cuda_stream, stats=False)
            assert rc == 0
    c.two_steps()
    for _ in range(2):
        x.copy_(c.start)
        g.replay()
        c.check(x, 1)
        c.check(y, 0)
        c.two_steps()
    # direct steps on the caller's own stream
    with torch.cuda.stream(s):
        x.copy_(c.start)
        for src, dst in ((x, y), (y, x)):
            assert c.call(src, dst, c.H.GLOBAL_CFL, 0.5, s.cuda_stream, stats=False)[0] == 0
    c.check(x, 1)


if __name__ == "__main__":
    sys.path[:0] = [os.path.dirname(HERE), os.path.join(os.path.dirname(HERE), "oracle"), HERE]
    {"after_refused": _after_refused, "captured": _captured}[sys.argv[1]]()
