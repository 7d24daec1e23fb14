"""The solve loops' early exit: a kernel whose blocks start late, since other work holds the SMs, stops,
pauses or goes on as a whole, so a solve has the same bits on a busy GPU as on an idle one: the mixed
solve (which pauses a dozen times), and solves of indefinite systems, which end in a breakdown, one
by one and as members of a batch of several waves of blocks."""
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


class Busy:
    """Other work on the GPU while the body runs."""

    def __enter__(self):
        import torch
        a = torch.randn(2048, 2048, device="cuda")
        torch.cuda.synchronize()
        self.stop = threading.Event()

        def load():
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                while not self.stop.is_set():
                    for _ in range(20):
                        torch.sin(a @ a)
                    s.synchronize()

        self.t = threading.Thread(target=load)
        self.t.start()

    def __exit__(self, *exc):
        self.stop.set()
        self.t.join()


@pytest.mark.parametrize("kind", ["mixed", "fp64", "ssor"])
def test_same_bits_on_a_busy_gpu(fb, kind):
    import torch
    solve, breaks = solver(fb, kind)
    x, conv, its, res, brk = solve()
    assert bool(brk) == breaks and bool(conv) != breaks
    with Busy():
        runs = [solve() for _ in range(8)]
    for y, _, it, _, b in runs:
        assert torch.equal(y, x) and it == its and b == brk


@pytest.mark.parametrize("mixed", [False, True])
def test_members_of_a_batch(fb, mixed):
    import torch
    mats = [indefinite(fb, n) for n in (200001, 300, 5003, 90001)]
    mats.insert(1, build(fb, "helmholtz_sin", 60, 2)["K"])
    for K in mats:
        fb.JacobiPreconditioner(K)
    rhs = [torch.as_tensor(np.random.default_rng(i).standard_normal(K.nrows)).cuda() for i, K in enumerate(mats)]
    B = fb.Batch(mats)
    xs, res = B.solve(rhs, tol=1e-10, mixed=mixed, engine="lockstep")
    assert res[1]["converged"] and not res[1]["breakdown"]
    assert all(r["breakdown"] and not r["converged"] for i, r in enumerate(res) if i != 1)
    ref = [x.clone() for x in xs]
    with Busy():
        for _ in range(5):
            ys, again = B.solve(rhs, tol=1e-10, mixed=mixed, engine="lockstep")
            assert all(torch.equal(x, y) for x, y in zip(ref, ys))
            assert [r["iterations"] for r in again] == [r["iterations"] for r in res]
