"""The solve loops' early exit: a kernel whose blocks start late, since other work holds the SMs, stops,
pauses or goes on as a whole, so a solve has the same bits on a busy GPU as on an idle one: the mixed
solve (which pauses a dozen times), and solves of indefinite systems, which end in a breakdown."""
import threading

import numpy as np
import pytest
import scipy.sparse as sp

from gpu_problems import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


def indefinite(fb, n):
    """Seven entries a row, one row in 97 with a negative diagonal."""
    rng = np.random.default_rng(11)
    B = sp.diags([rng.uniform(-1, 0, n) for _ in range(3)], [1, 2, 40], shape=(n, n)).tocsr()
    B = B + B.T
    d = 1.5 * np.asarray(abs(B).sum(axis=1)).ravel() + 1.0
    d[::97] *= -1.0
    A = sp.csr_matrix(B + sp.diags(d))
    A.sort_indices()
    return fb.CSRMatrix.from_arrays(n, n, A.indptr, A.indices, A.data)


def solver(fb, kind):
    """A function that solves anew, and whether it breaks down."""
    import torch
    if kind == "mixed":
        pr = build(fb, "helmholtz_sin", 150, 2)
        M = fb.JacobiPreconditioner(pr["K"])
        return lambda: fb.cg_solve(pr["K"], M, pr["rhs"], None, 100000, 1e-11, mixed=True), False
    n = 3001 if kind == "ssor" else 330001
    K = indefinite(fb, n)
    b = torch.as_tensor(np.random.default_rng(1).standard_normal(n)).cuda()
    M = fb.SSORPreconditioner(K, 1.2) if kind == "ssor" else None
    return lambda: fb.cg_solve(K, M, b, None, 1000, 1e-11), True


@pytest.mark.parametrize("kind", ["mixed", "fp64", "ssor"])
def test_same_bits_on_a_busy_gpu(fb, kind):
    import torch
    solve, breaks = solver(fb, kind)
    x, conv, its, res, brk = solve()
    assert bool(brk) == breaks and bool(conv) != breaks
    a = torch.randn(2048, 2048, device="cuda")
    torch.cuda.synchronize()
    stop = threading.Event()

    def load():
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            while not stop.is_set():
                for _ in range(20):
                    torch.sin(a @ a)
                s.synchronize()

    t = threading.Thread(target=load)
    t.start()
    try:
        runs = [solve() for _ in range(8)]
    finally:
        stop.set()
        t.join()
    for y, _, it, _, b in runs:
        assert torch.equal(y, x) and it == its and b == brk
