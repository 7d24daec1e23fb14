"""The FP32 row sums of the mixed solve, by a system that shows them: a row's 33 terms are 1 - 15 u (the
row sum), sixteen small ones before it and sixteen after it, each just under half an ulp of the sum, so
one chain in entry order loses the last sixteen (15 u).  Sums of four chains and a tree, which both
forms of the SpMV are to be, keep them."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu

U = 2.0 ** -24            # FP32's unit roundoff


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


# a term passes through ceil(33 / 4) additions of its chain and 2 of the tree; alpha and x are rounded
# once each, and the terms' sum of magnitudes is the sum itself (to 1e-6)
BOUND = (9 + 2 + 2) * U


@pytest.mark.parametrize("form", ["slices", "lane groups"])
def test_row_sums(fb, form):
    import torch
    n, c = 2048, 30 / 32 * 2.0 ** -25
    offsets = list(range(1, 32, 2))
    A = sp.diags([np.full(n - o, -c) for o in offsets], offsets, shape=(n, n))
    A = sp.csr_matrix(A + A.T + sp.identity(n))
    A.sort_indices()
    K = fb.CSRMatrix.from_arrays(n, n, A.indptr, A.indices, A.data)
    if form == "lane groups":
        K.set_spmv_tpr(4 | 1 << 8)
    M = fb.JacobiPreconditioner(K)
    b = np.where(np.arange(n) % 2 == 0, 1.0, -1.0)
    x = fb.cg_solve(K, M, torch.as_tensor(b).cuda(), None, 1, 1e-14, mixed=True)[0].cpu().numpy()
    alpha = (b @ b) / (b @ (A @ b))                      # the first step of CG with D = I
    assert np.abs(x / (alpha * b) - 1.0).max() <= BOUND
