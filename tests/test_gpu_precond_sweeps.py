"""The level sweeps of ILU(0) and SSOR (csrc/precond.cu) against the same arithmetic done row by row
on the host, bit for bit: one level of all rows (read where it lies), a level a row, levels wider
than the block, rows longer than what is loaded ahead, z in and out of shared memory."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


def ilu0(ip, ix, v):
    """The reference's IKJ elimination; Python floats round every operation once, as the kernel does."""
    v = [float(t) for t in v]
    n = len(ip) - 1
    row = [{int(ix[q]): q for q in range(ip[i], ip[i + 1])} for i in range(n)]
    for i in range(n):
        for p in range(ip[i], row[i][i]):
            k = int(ix[p])
            v[p] /= v[row[k][k]]
            for q in range(row[k][k] + 1, ip[k + 1]):
                s = row[i].get(int(ix[q]))
                if s is not None:
                    v[s] -= v[p] * v[q]
    return v


def sweeps(ip, ix, v, r, w=None):
    n = len(ip) - 1
    d = [ip[i] + int(np.searchsorted(ix[ip[i]:ip[i + 1]], i)) for i in range(n)]
    z = [float(t) for t in r]
    for i in range(n):
        s = z[i]
        for p in range(ip[i], d[i]):
            s -= v[p] * z[ix[p]]
        z[i] = s if w is None else s * w / v[d[i]]
    if w is not None:
        c = (2.0 - w) / w
        z = [z[i] * (c * v[d[i]] / w) for i in range(n)]
    for i in reversed(range(n)):
        s = z[i]
        for p in range(d[i] + 1, ip[i + 1]):
            s -= v[p] * z[ix[p]]
        z[i] = s / v[d[i]] if w is None else s * w / v[d[i]]
    return np.array(z)


def matrix(kind):
    rng = np.random.default_rng(7)
    if kind == "diagonal":
        return sp.diags(rng.uniform(1, 2, 30000))
    if kind == "chain":
        n = 700
        return sp.diags([np.full(n - 1, -0.3), rng.uniform(1, 2, n), np.full(n - 1, -0.4)], [-1, 0, 1])
    if kind == "one":
        return sp.csr_matrix(np.array([[3.0]]))
    if kind == "arrow":
        n = 500
        A = sp.lil_matrix((n, n))
        A.setdiag(rng.uniform(2, 3, n))
        A[0, 1:] = rng.uniform(-1e-3, 1e-3, n - 1)
        A[1:, 0] = rng.uniform(-1e-3, 1e-3, n - 1)[:, None]
        return A
    n, per = {"random": (3000, 4), "dense rows": (400, 30), "wide": (40000, 1)}[kind]
    i = np.repeat(np.arange(n), per)
    B = sp.csr_matrix((rng.uniform(-1, 1, n * per), (i, rng.integers(0, n, n * per))), shape=(n, n))
    B = B + B.T
    return B + sp.diags(2.0 + np.asarray(abs(B).sum(axis=1)).ravel())


@pytest.mark.parametrize("kind", ["one", "diagonal", "chain", "arrow", "random", "dense rows", "wide"])
def test_sweeps_bit_exact(fb, kind):
    A = sp.csr_matrix(matrix(kind))
    A.sum_duplicates()
    A.sort_indices()
    K = fb.CSRMatrix.from_arrays(A.shape[0], A.shape[0], A.indptr, A.indices, A.data)
    r = np.random.default_rng(1).standard_normal(A.shape[0])
    r[::5] = -0.0
    v = ilu0(A.indptr, A.indices, A.data)
    got = fb.ILU0Preconditioner(K).apply(r).cpu().numpy()
    want = sweeps(A.indptr, A.indices, v, r)
    assert np.array_equal(got.view(np.int64), want.view(np.int64))
    got = fb.SSORPreconditioner(K, 1.3).apply(r).cpu().numpy()
    want = sweeps(A.indptr, A.indices, [float(t) for t in A.data], r, 1.3)
    assert np.array_equal(got.view(np.int64), want.view(np.int64))
