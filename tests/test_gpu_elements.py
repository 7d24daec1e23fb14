"""The element-tensor paths of the FAST assembly (csrc/assemble.cu: varying coefficients, constant
forms without symmetric pairs, load vectors) against the EXACT mode, which is pinned to the
reference bit for bit, on a mesh with moved vertices.

Tolerance: an entry is a sum of at most 8 cells x 4 terms x 36 points products, each formed with
about 8 roundings: 1152 x 8 x 1.1e-16 = 1e-12 of the largest contribution at worst.  That is the
largest entry, or, where a whole matrix cancels (one unknown, test times derivative: the sum is 0
and EXACT leaves -3e-17), a cell's integral: cell area h^2 / 2 times a value or derivative of order
h^-(orders)."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
PI = math.pi


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


def space(fb, N, k):
    m = fb.rectangle_mesh(0, 0, 1, 1, N, N)
    pts = m.points.copy()
    inner = ((pts > 0) & (pts < 1)).all(axis=1)
    pts[inner] += np.random.default_rng(N).uniform(-0.2 / N, 0.2 / N, (int(inner.sum()), 2))
    return fb.LagrangeSpace2D(fb.Mesh2D(pts, m.tris), k, bc="dirichlet")


def coefs(fb, V, Q):
    import torch
    rng = np.random.default_rng(3)
    dev = lambda a: torch.as_tensor(a).cuda()
    return dict(one=fb.Coef.const(1.0), two=fb.Coef.const(-2.5), sin=fb.Coef.sinsin(1.0, 0.5, 2 * PI, 3 * PI),
                helm=fb.Coef.helmholtz_sinsin(3.0, PI, 2 * PI), field=fb.Coef.field(dev(rng.standard_normal(V.dim))),
                points=fb.Coef.points(dev(rng.uniform(0.5, 2.0, V.mesh.ncells * Q.nq))))


MATRICES = [([0], [1], ["one"]),                                        # two unsymmetric pairs
            ([0, 1], [2, 0], ["one", "two"]),
            ([1, 2], [1, 2], ["sin", "sin"]),                           # one coefficient in two terms
            ([1, 2, 0], [1, 2, 0], ["sin", "points", "one"]),
            ([0, 0, 1, 2], [0, 1, 2, 0], ["field", "helm", "two", "points"]),
            ([0], [0], ["points"])]
VECTORS = [([0], ["one"]), ([0], ["sin"]), ([1, 2], ["helm", "field"]), ([0, 1, 0, 2], ["one", "points", "field", "one"])]


# one cell pair, sizes around a block of cells and of rows, and a mesh of several blocks
@pytest.mark.parametrize("N,k", [(2, 1), (8, 1), (9, 2), (16, 1), (7, 3), (30, 2), (5, 4), (3, 5)])
def test_elements_match_exact(fb, N, k):
    V = space(fb, N, k)
    Q = V.cache(2 * k + 1)
    P = V.pattern()
    c = coefs(fb, V, Q)
    def close(x, ref, orders):
        return np.all(np.abs(x - ref) <= 1e-12 * max(np.abs(ref).max(), 0.5 * N ** -(2.0 - orders)))

    for a, b, names in MATRICES:
        out = []
        for exact in (True, False):
            K = fb.CSRMatrix(P)
            fb.assemble_matrix_2d(Q, Q, a, b, [c[t] for t in names], K, exact=exact, jacobi=False)
            out.append(K.data)
        assert close(out[1], out[0], min((i > 0) + (j > 0) for i, j in zip(a, b))), (a, b, names)
    for a, names in VECTORS:
        ref = fb.assemble_vector_2d(Q, a, [c[t] for t in names], P, exact=True).cpu().numpy()
        assert close(fb.assemble_vector_2d(Q, a, [c[t] for t in names], P).cpu().numpy(), ref, min(i > 0 for i in a)), (a, names)
