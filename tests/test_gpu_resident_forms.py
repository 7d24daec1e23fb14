"""Which form of the on-chip solve takes a system (csrc/resident.cu, resident_plan): few entries a row and
more rows than a cluster keeps go to the grid, and so do rows of very uneven length that a cluster's
block turns out not to hold.  Told by the launches of a solve: one on chip, three an iteration else."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


def tridiagonal(n):
    e = np.full(n - 1, -1.0)
    return sp.diags([e, np.full(n, 2.2), e], [-1, 0, 1])


def uneven(n, heavy):
    """Diagonal but for the last `heavy` rows, which have 60 entries among themselves."""
    rng = np.random.default_rng(1)
    i = np.repeat(np.arange(n - heavy, n), 30)
    B = sp.csr_matrix((rng.uniform(-1, 1, i.size), (i, rng.integers(n - heavy, n, i.size))), shape=(n, n))
    B = B + B.T
    return B + sp.diags(1.2 * np.asarray(abs(B).sum(axis=1)).ravel() + rng.uniform(1, 2, n))


@pytest.mark.parametrize("kind,n", [("tridiagonal", 32768), ("tridiagonal", 32769), ("tridiagonal", 60000), ("uneven", 26000)])
def test_on_chip(fb, kind, n):
    A = sp.csr_matrix(tridiagonal(n) if kind == "tridiagonal" else uneven(n, 1000))
    A.sort_indices()
    K = fb.CSRMatrix.from_arrays(n, n, A.indptr, A.indices, A.data)
    M = fb.JacobiPreconditioner(K)
    xd = np.random.default_rng(2).standard_normal(n)
    fb.cg_solve(K, M, A @ xd, None, 1000, 1e-12)          # a form that does not fit is found here
    before = fb.lib.femd_cuda_kernel_launches()
    x, conv, its, res, brk = fb.cg_solve(K, M, A @ xd, None, 1000, 1e-12)
    launches = fb.lib.femd_cuda_kernel_launches() - before
    assert conv and not brk and its >= 10 and launches <= 3
    # condition numbers below 30
    assert np.linalg.norm(x.cpu().numpy() - xd) <= 1e-10 * np.linalg.norm(xd)


def test_a_shape_set_by_hand_is_kept_to(fb):
    n = 5000
    A = sp.csr_matrix(tridiagonal(n))
    K = fb.CSRMatrix.from_arrays(n, n, A.indptr, A.indices, A.data)
    M = fb.JacobiPreconditioner(K)
    xd = np.random.default_rng(2).standard_normal(n)

    def solve():
        before = fb.lib.femd_cuda_kernel_launches()
        x, conv, its, res, brk = fb.cg_solve(K, M, A @ xd, None, 1000, 1e-12)
        assert conv and np.linalg.norm(x.cpu().numpy() - xd) <= 1e-10 * np.linalg.norm(xd)
        return fb.lib.femd_cuda_kernel_launches() - before

    assert solve() <= 3
    K.set_spmv_tpr(4 | 1 << 8)
    assert solve() > 30
    K.set_spmv_tpr(0)
    assert solve() <= 3
    K.autotune_spmv(True)
    assert solve() <= 3
