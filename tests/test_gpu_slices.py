"""The sliced SpMV of the streaming solves (csrc/krylov.cu): systems past the on-chip solve against
known solutions, and the solve that keeps nothing (whose sums come from the CSR) bit for bit;
rows not a multiple of the slices, uneven rows that fill the slices too much, rows longer than a
warp's shared memory, FP32 values."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from gpu_problems import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


def system(fb, kind):
    """A matrix past the on-chip solve's room, as a CSRMatrix and on the host."""
    rng = np.random.default_rng(5)
    if kind in ("p1", "p2", "p3"):
        N, k = {"p1": (601, 1), "p2": (260, 2), "p3": (131, 3)}[kind]
        pr = build(fb, "helmholtz_sin", N, k, c=1.0)
        K = pr["K"]
        ip, ix = pr["P"].to_host()
        return K, sp.csr_matrix((K.data, ix, ip), shape=(K.nrows, K.nrows))
    n = 330001
    if kind == "band":                        # even rows, 7 entries
        B = sp.diags([rng.uniform(-1, 0, n) for _ in range(3)], [1, 2, 40], shape=(n, n)).tocsr()
    else:                                     # uneven rows: one in 50 couples to 60 others, one to 1000
        i = np.repeat(np.arange(0, n, 50), 60)
        i = np.concatenate([i, np.full(1000, 7)])
        j = rng.integers(0, n, i.size)
        B = sp.csr_matrix((rng.uniform(-1, 0, i.size), (i, j)), shape=(n, n))
    B = B + B.T
    A = sp.csr_matrix(B + sp.diags(1.5 * np.asarray(abs(B).sum(axis=1)).ravel() + 1.0))
    A.sort_indices()
    return fb.CSRMatrix.from_arrays(n, n, A.indptr, A.indices, A.data), A


# relative residual 1e-12; condition numbers (Jacobi-scaled) below 1e5 for the meshes, 10 for the rest
@pytest.mark.parametrize("kind,bound", [("p1", 1e-8), ("p2", 1e-8), ("p3", 1e-8), ("band", 1e-11), ("uneven", 1e-11)])
def test_solves(fb, kind, bound):
    import torch
    from femd_b200 import _native as N
    K, A = system(fb, kind)
    n = K.nrows
    assert 10.0 * K.nnz + 4.0 * n > 141 * 1024 * 148 or n > 320000       # not solved on chip
    x = np.random.default_rng(2).standard_normal(n)
    b = torch.as_tensor(A @ x).cuda()
    M = fb.JacobiPreconditioner(K)
    got, conv, its, res, brk = fb.cg_solve(K, M, b, None, 100000, 1e-12)
    assert conv and not brk and res <= 1.1e-12
    assert np.linalg.norm(got.cpu().numpy() - x) <= bound * np.linalg.norm(x)
    # the values changed: the next solve takes the new ones
    K.set_data(2.0 * K.data)
    M = fb.JacobiPreconditioner(K)
    half = fb.cg_solve(K, M, b, None, 100000, 1e-12)[0]
    assert np.linalg.norm(2.0 * half.cpu().numpy() - x) <= bound * np.linalg.norm(x)
    # the same bits from the solve that allocates nothing
    y = torch.zeros_like(b)
    r = N.femd_cg_result()
    ctx = K.ctx
    ctx.enter()
    N.check(fb.lib.femd_cuda_cg_jacobi_noalloc(ctx.h, K.h, 1, b.data_ptr(), y.data_ptr(), 100000, 1e-12, C.byref(r)))
    ctx.leave()
    assert torch.equal(y, half) and r.iterations == N.femd_cg_result.from_buffer_copy(fb.cg_solve.last).iterations
    # FP32 inner iteration
    mixed, conv, its, res, brk = fb.cg_solve(K, M, b, None, 100000, 1e-12, mixed=True)
    assert conv and not brk
    assert np.linalg.norm(2.0 * mixed.cpu().numpy() - x) <= bound * np.linalg.norm(x)
    # a chosen lane-group shape is kept to
    K.set_spmv_tpr(4 | 4 << 8)
    again = fb.cg_solve(K, M, b, None, 100000, 1e-12)[0]
    assert np.linalg.norm((again - half).cpu().numpy()) <= bound * np.linalg.norm(x)


def test_a_tuned_shape_leaves_the_slices(fb):
    """The autotuner's shape is for products: the solve keeps the slices, and so its bits."""
    import torch
    K, A = system(fb, "band")
    b = torch.as_tensor(np.random.default_rng(3).standard_normal(K.nrows)).cuda()
    M = fb.JacobiPreconditioner(K)
    x = fb.cg_solve(K, M, b, None, 1000, 1e-10)[0]
    shape, us = K.autotune_spmv(True)
    assert shape != 0 and us > 0.0
    assert torch.equal(fb.cg_solve(K, M, b, None, 1000, 1e-10)[0], x)
