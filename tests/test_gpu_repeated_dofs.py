"""Cells that name a dof twice (a mesh one cell wide with its sides identified): the assembly adds
all their contributions, G^T A G with A the matrix before the sides are identified.

Tolerance: an entry is a sum of at most 8 cells x 9 repeats x 3 terms x 36 points products, each formed
with about 8 roundings: 7776 x 8 x 1.1e-16 < 1e-11 of the largest contribution, an entry of A (G^T A G
may cancel: value times derivative at P1 is 0)."""
import ctypes as C
import math

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu
PI = math.pi


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


def pattern(fb, n, dofs):
    import torch
    from femd_b200 import _native as N
    ctx = fb.context()
    d = torch.as_tensor(np.ascontiguousarray(dofs, dtype=np.int32)).cuda()
    h = C.c_void_p()
    ctx.enter()
    N.check(fb.lib.femd_cuda_pattern_from_cells(ctx.h, n, dofs.shape[0], dofs.shape[1], C.c_void_p(d.data_ptr()), C.byref(h)))
    P = fb.SparsityPattern(h, ctx)
    P.ncells, P.nloc = dofs.shape
    return P


@pytest.mark.parametrize("exact", [False, True])
@pytest.mark.parametrize("form", ["constant", "varying", "unsymmetric"])
@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_all_are_added(fb, k, form, exact):
    m = fb.rectangle_mesh(0, 0, 1, 1, 1, 9)
    V = fb.LagrangeSpace2D(m, k)
    # the vertices of the side x = 1 become those of x = 0
    dofs, at = np.array(V.cell_dofs), {}
    for cell, tri in zip(dofs, m.tris):
        at.update({int(v): int(d) for v, d in zip(tri, cell)})
    glue = np.arange(V.dim)
    for v, d in at.items():
        if m.points[v, 0] == 1.0:
            glue[d] = at[int(np.flatnonzero((m.points[:, 0] == 0.0) & (m.points[:, 1] == m.points[v, 1]))[0])]
    dofs = glue[dofs]
    assert any(len(set(d)) < len(d) for d in dofs)
    P = pattern(fb, V.dim, dofs)
    Q = V.cache(2 * k + 1)
    one, sin = fb.Coef.const(1.0), fb.Coef.sinsin(1.0, 0.5, 2 * PI, 3 * PI)
    a, b, c = {"constant": ([1, 2, 0], [1, 2, 0], [one] * 3), "varying": ([1, 2], [1, 2], [sin] * 2),
               "unsymmetric": ([0], [1], [one])}[form]
    def assembled(P):
        K = fb.CSRMatrix(P)
        fb.assemble_matrix_2d(Q, Q, a, b, c, K, jacobi=False, exact=exact)
        ip, ix = P.to_host()
        return sp.csr_matrix((K.data, ix, ip), shape=(V.dim, V.dim))

    G = sp.csr_matrix((np.ones(V.dim), (np.arange(V.dim), glue)), shape=(V.dim, V.dim))
    A = assembled(V.pattern())
    want = (G.T @ A @ G).toarray()
    assert np.abs(assembled(P).toarray() - want).max() <= 1e-11 * np.abs(A.data).max()
