"""The chunks of ILU(0)'s and SSOR's sweeps (csrc/precond_host.h), on the host: every row once, after the
rows it reads, no chunk of two levels, none larger than the limit; a level of more bytes than 32-bit
places reach is several chunks; and, on a GPU, such a level's sweeps."""
import ctypes as C

import numpy as np
import pytest
import scipy.sparse as sp

from femd_b200 import _native as N


def chunks(A, forward, limit):
    A = sp.csr_matrix(A)
    A.sort_indices()
    n, ip, ix = A.shape[0], A.indptr.astype(np.int32), A.indices.astype(np.int32)
    count = C.c_int()
    N.check(N.lib.femd_host_precond_chunks(n, ip.ctypes.data, ix.ctypes.data, int(forward), limit, C.byref(count), None, None, None))
    rows, first, size = np.empty(n, np.int32), np.empty(count.value + 1, np.int32), np.empty(count.value, np.int64)
    N.check(N.lib.femd_host_precond_chunks(n, ip.ctypes.data, ix.ctypes.data, int(forward), limit, C.byref(count),
                                           rows.ctypes.data, first.ctypes.data, size.ctypes.data))
    return A, rows, first, size


def matrix(kind):
    rng = np.random.default_rng(3)
    if kind == "diagonal":
        return sp.identity(5000)
    n, per = {"random": (1500, 3), "dense rows": (300, 20)}[kind]
    i = np.repeat(np.arange(n), per)
    B = sp.csr_matrix((rng.uniform(0.1, 1, n * per), (i, rng.integers(0, n, n * per))), shape=(n, n))
    if kind == "dense rows":
        B = B + sp.csr_matrix((np.ones(n), (np.full(n, 7), np.arange(n))), shape=(n, n))
    return B + B.T + sp.identity(n)


@pytest.mark.parametrize("limit", [0, 700, 4096, 20000])
@pytest.mark.parametrize("forward", [True, False])
@pytest.mark.parametrize("kind", ["diagonal", "random", "dense rows"])
def test_order(kind, forward, limit):
    A, rows, first, size = chunks(matrix(kind), forward, limit)
    n = A.shape[0]
    assert first[0] == 0 and first[-1] == n and np.array_equal(np.sort(rows), np.arange(n))
    chunk = np.empty(n, np.int64)
    chunk[rows] = np.repeat(np.arange(size.size), np.diff(first))
    level = np.zeros(n, np.int64)
    for i in range(n) if forward else reversed(range(n)):
        c = A.indices[A.indptr[i]:A.indptr[i + 1]]
        c = c[c < i] if forward else c[c > i]
        assert (chunk[c] < chunk[i]).all()
        level[i] = level[c].max(initial=-1) + 1
    assert all(np.unique(level[rows[a:b]]).size == 1 for a, b in zip(first[:-1], first[1:]))
    assert (np.diff(first) > 0).all() and (size % 16 == 0).all()
    if limit == 0:
        assert size.size == level.max(initial=-1) + 1
    else:
        assert ((size <= limit) | (np.diff(first) <= 8)).all()


def test_places_fit_32_bits():
    n = 70_000_000                                        # one level of 2.24 GB of records
    ip, ix = np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32)
    count = C.c_int()
    size = np.empty(64, np.int64)
    N.check(N.lib.femd_host_precond_chunks(n, ip.ctypes.data, ix.ctypes.data, 1, 0, C.byref(count), None, None, size.ctypes.data))
    assert 1 < count.value <= size.size                   # at least 1 GB - a warp's rows each
    assert size[:count.value].max() < 2 ** 31 and size[:count.value].sum() >= 32 * n


@pytest.mark.gpu
def test_a_level_of_several_chunks():
    import torch
    import femd_b200 as fb
    n = 34_000_000                                        # 1.09 GB of records: two chunks each way
    d = np.random.default_rng(0).uniform(1.0, 2.0, n)
    K = fb.CSRMatrix.from_arrays(n, n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), d)
    M = fb.ILU0Preconditioner(K)
    assert M.levels == (1, 1)
    r = torch.as_tensor(np.random.default_rng(1).standard_normal(n)).cuda()
    assert torch.equal(M.apply(r), r / torch.as_tensor(d).cuda())
