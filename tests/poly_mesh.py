"""A mesh of cells with three to eight faces, for the tests of the widest kernel variants.

Rows of a jittered node grid on [0, 2] x [0, 1] are cut into runs of one, two or three squares (4, 6
and 8 faces), each longer by a triangle in some (5 and 7 faces, the triangle's other half a cell of
its own).  Colours 1-4: bottom, right, top, left.  Duck-types Mesh for Solver and the oracle.
"""
import ctypes as ct

import numpy as np

from cfd_optimisations_b200 import native as N


def _row(nx, j):
    """Cells of row j as loops of (i, j) nodes."""
    kinds = [("run", 1), ("run", 2), ("run", 3), ("cut", 1), ("cut", 2)]
    i, k, cells = 0, j, []
    while i < nx:
        kind, w = kinds[k % len(kinds)]
        k += 1
        need = w + (kind == "cut")
        if i + need > nx:
            kind, w, need = "run", 1, 1
        bottom = [(a, j) for a in range(i, i + need + 1)]
        if kind == "run":
            cells.append(bottom + [(a, j + 1) for a in range(i + w, i - 1, -1)])
        else:
            cells.append(bottom + [(a, j + 1) for a in range(i + w, i - 1, -1)])
            cells.append([(i + need, j), (i + need, j + 1), (i + w, j + 1)])
        i += need
    return cells


class PolyMesh:
    def __init__(self, nx: int, ny: int, seed: int = 1):
        r = np.random.default_rng(seed)
        X, Y = np.meshgrid(np.linspace(0, 2, nx + 1), np.linspace(0, 1, ny + 1))
        jig = 0.1 * np.array([2 / nx, 1 / ny])
        inner = np.zeros(X.shape, dtype=bool)
        inner[1:-1, 1:-1] = True
        X = X + np.where(inner, jig[0] * r.uniform(-1, 1, X.shape), 0)
        Y = Y + np.where(inner, jig[1] * r.uniform(-1, 1, X.shape), 0)
        nid = lambda p: p[1] * (nx + 1) + p[0]
        cells = [[nid(p) for p in c] for j in range(ny) for c in _row(nx, j)]
        cells = [cells[k] for k in r.permutation(len(cells))]          # neighbours far apart in the input order
        edges = {}
        for c, loop in enumerate(cells):
            for a, b in zip(loop, loop[1:] + loop[:1]):
                edges.setdefault((min(a, b), max(a, b)), []).append(c)
        interior = [(e, cs) for e, cs in edges.items() if len(cs) == 2]
        side = lambda e: (0 if e[0] <= nx and e[1] <= nx else 1 if e[0] % (nx + 1) == e[1] % (nx + 1) == nx
                          else 2 if e[0] >= ny * (nx + 1) else 3)
        boundary = sorted(((side(e), e, cs[0]) for e, cs in edges.items() if len(cs) == 1))
        fn = [e for e, _ in interior] + [e for _, e, _ in boundary]
        fc = [(min(cs), max(cs)) for _, cs in interior] + [(c, len(cells) + k) for k, (_, _, c) in enumerate(boundary)]
        cn = cells + [list(e) for _, e, _ in boundary]                 # ghosts: their face's two nodes
        count = np.bincount([s for s, _, _ in boundary], minlength=4)
        coloff = np.concatenate([[0], len(interior) + np.concatenate([[0], np.cumsum(count)])])
        i32 = lambda x: np.ascontiguousarray(x, dtype=np.int32)
        self._a = dict(dim=2, Nn=X.size, Ncol=5, NBCcol=4, Nc=len(cn), Nf=len(fn), coltag=i32([0, 1, 2, 3, 4]),
                       coloff=i32(coloff), nodes=np.column_stack([X.ravel(), Y.ravel()]).ravel().copy(),
                       fn_con=i32(fn).ravel(), fc_con=i32(fc).ravel(),
                       cn_off=i32(np.concatenate([[0], np.cumsum([len(c) for c in cn])])),
                       cn_con=i32(np.concatenate(cn)))
        self.Nc, self.Nf = len(cn), len(fn)

    def arrays(self):
        return dict(self._a)

    def view(self):
        a = self._a
        i = lambda k: a[k].ctypes.data_as(N._ip)
        return N.MeshView(2, a["Nn"], a["Ncol"], a["NBCcol"], a["Nc"], a["Nf"], i("coltag"), i("coloff"),
                          a["nodes"].ctypes.data_as(ct.POINTER(ct.c_double)), i("fn_con"), i("fc_con"), i("cn_off"),
                          i("cn_con"), None, None)
