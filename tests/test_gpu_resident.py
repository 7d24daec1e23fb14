"""The on-chip Jacobi-PCG (csrc/resident.cu) behind cg_solve: against known solutions at the edges of
its layout (fewer rows than blocks, one lane or several a row, both forms of its sums, rows that
do not fit and go to the streaming loop) and at the edges of the stopping rule."""
import numpy as np
import pytest
import scipy.sparse as sp

from gpu_problems import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


def from_scipy(fb, A):
    A = sp.csr_matrix(A)
    A.sort_indices()
    return fb.CSRMatrix.from_arrays(A.shape[0], A.shape[1], A.indptr, A.indices, A.data)


def spd(n, per_row, seed):
    """A diagonally dominant matrix with random couplings (condition number below 10)."""
    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), per_row)
    j = rng.integers(0, n, n * per_row)
    B = sp.csr_matrix((rng.uniform(-1, 1, n * per_row), (i, j)), shape=(n, n))
    B = B + B.T
    off = np.asarray(abs(B).sum(axis=1)).ravel()
    return sp.csr_matrix(B + sp.diags(1.2 * off + 1.0))


def check(fb, A, K, jac, x0, seed, bound):
    rng = np.random.default_rng(seed)
    n = A.shape[0]
    xd = rng.standard_normal(n)
    b = A @ xd
    M = fb.JacobiPreconditioner(K) if jac else None
    start = rng.standard_normal(n) if x0 else None
    x, conv, its, res, brk = fb.cg_solve(K, M, b, start, 100000, 1e-12)
    x = x.cpu().numpy()
    assert conv and not brk and res <= 1.1e-12
    assert np.linalg.norm(x - xd) <= bound * np.linalg.norm(xd)
    y = fb.cg_solve(K, M, b, start, 100000, 1e-12)[0].cpu().numpy()
    assert np.array_equal(x, y)


# the relative residual is 1e-12 and the Jacobi-scaled condition numbers are below 1e4 (N k <= 120):
# 1e-8 relative in x.  N = 2..4: blocks without rows; 150 P2 and 80 P3: past the cluster
@pytest.mark.parametrize("N,k,jac,x0", [(2, 1, True, False), (3, 1, False, True), (4, 2, True, True), (21, 3, True, False),
                                        (37, 2, False, False), (64, 1, True, True), (95, 1, True, False), (60, 2, True, False),
                                        (40, 3, False, True)])
def test_meshes(fb, N, k, jac, x0):
    pr = build(fb, "poisson_vec", N, k, c=1.0, b_vec=np.zeros(1))
    ip, ix = pr["P"].to_host()
    K = pr["K"]
    check(fb, sp.csr_matrix((K.data, ix, ip), shape=(K.nrows, K.nrows)), K, jac, x0, N, 1e-8)


# condition numbers below 10: 1e-11 relative.  Random columns (every entry another halo place), rows
# of one entry and of hundreds, and systems whose blocks cannot hold them (320,000 rows: over the
# rows a block keeps; 60,000 x 100 random columns: over its halo)
@pytest.mark.parametrize("n,per_row", [(1, 0), (17, 3), (500, 40), (5000, 3), (30000, 6), (60000, 50), (310000, 0), (320000, 0)])
def test_general_matrices(fb, n, per_row):
    A = spd(n, per_row, n) if per_row else sp.diags(np.random.default_rng(n).uniform(1, 5, n)).tocsr()
    check(fb, A, from_scipy(fb, A), True, n % 2 == 0, n, 1e-11)


def test_long_row(fb):
    """An arrow matrix: one row and one column full."""
    n = 9000
    A = sp.lil_matrix((n, n))
    A.setdiag(4.0)
    A[0, 1:] = 0.01
    A[1:, 0] = 0.01
    A[0, 0] = 4.0 + 0.0001 * n
    A = A.tocsr()
    check(fb, A, from_scipy(fb, A), True, False, 5, 1e-10)


@pytest.mark.parametrize("N,k", [(6, 2), (100, 2)])
def test_stopping_rule(fb, N, k):
    import torch
    pr = build(fb, "poisson_vec", N, k, c=1.0, b_vec=np.zeros(1))
    K = pr["K"]
    n = K.nrows
    M = fb.JacobiPreconditioner(K)
    b = torch.as_tensor(np.random.default_rng(3).standard_normal(n)).cuda()
    # b = 0: x = 0 whatever the start
    x, conv, its, res, brk = fb.cg_solve(K, M, torch.zeros_like(b), torch.ones_like(b), 100, 1e-10)
    assert conv and its == 0 and res == 0.0 and not x.any()
    # a start within the tolerance: no iteration, x unchanged
    full = fb.cg_solve(K, M, b, None, 100000, 1e-13)[0]
    x, conv, its, res, brk = fb.cg_solve(K, M, b, full, 100000, 1e-10)
    assert conv and its == 0 and torch.equal(x, full)
    # stopped by max_iter; the residual is the true one
    x, conv, its, res, brk = fb.cg_solve(K, M, b, None, 3, 1e-10)
    assert its == 3 and not conv and not brk
    r = b - K.matvec(x)
    assert abs(float(r.norm() / b.norm()) - res) <= 1e-12 * res + 1e-15
    # an indefinite matrix: breakdown reported
    d = K.data.copy()
    K.set_data(-d)
    x, conv, its, res, brk = fb.cg_solve(K, None, b, None, 100, 1e-10)
    assert brk and not conv and its == 0
