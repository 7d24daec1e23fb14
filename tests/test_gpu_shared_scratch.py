"""What shares a context's scratch (assemblies, pattern builds, on-chip solves) used by several host
threads, and assemblies that a CUDA graph replays after the scratch has moved on: the same bits as
one call after another."""
import threading

import numpy as np
import pytest

from gpu_problems import PI

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


class Work:
    """Two matrices (cell factors, element matrices), a load and a solve on one space."""

    def __init__(self, fb, N, k):
        self.fb = fb
        self.V = fb.LagrangeSpace2D(fb.rectangle_mesh(0, 0, 1, 1, N, N), k, bc="dirichlet")
        self.Q, self.P = self.V.cache(2 * k + 1), self.V.pattern()
        self.K, self.L = fb.CSRMatrix(self.P), fb.CSRMatrix(self.P)
        one = fb.Coef.const(1.0)
        fb.assemble_matrix_2d(self.Q, self.Q, [1, 2, 0], [1, 2, 0], [one, one, one], self.K)
        self.coef = fb.Coef.sinsin(1.0, 0.5, 2 * PI, 3 * PI)
        import torch
        self.f = torch.zeros(self.V.dim, dtype=torch.float64, device="cuda")

    def assemble(self):
        fb, Q, one = self.fb, self.Q, self.fb.Coef.const(1.0)
        fb.assemble_matrix_2d(Q, Q, [1, 2, 0], [1, 2, 0], [one, one, one], self.K, jacobi=False)
        fb.assemble_matrix_2d(Q, Q, [1, 2], [1, 2], [self.coef, self.coef], self.L, jacobi=False)
        fb.assemble_vector_2d(Q, [0], [self.coef], self.P, out=self.f)

    def values(self):
        return [v.copy() for v in (self.K.data_tensor().cpu().numpy(), self.L.data_tensor().cpu().numpy(), self.f.cpu().numpy())]


def same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("k", [1, 2, 3])
def test_replayed_graph(fb, k):
    import torch
    w, other = Work(fb, 24, k), Work(fb, 40, k)
    w.assemble()
    ref = w.values()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=w.K.ctx.stream, capture_error_mode="thread_local"):
        w.assemble()
    for _ in range(2):
        other.V = fb.LagrangeSpace2D(fb.rectangle_mesh(0, 0, 1, 1, 90, 90), k, bc="dirichlet")
        other.V.pattern()                                # writes the scratch, and moves it
        other.assemble()
        for t in (w.K.data_tensor(), w.L.data_tensor(), w.f):
            t.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert same(w.values(), ref)


def test_threads_on_one_context(fb):
    import torch
    works = [Work(fb, N, k) for N, k in ((21, 2), (40, 1), (70, 3), (16, 3))]
    rhs = [torch.as_tensor(np.random.default_rng(i).standard_normal(w.V.dim)).cuda() for i, w in enumerate(works)]
    refs = []
    for w, b in zip(works, rhs):
        w.assemble()
        x, _, its, _, _ = fb.cg_solve(w.K, None, b, None, 5000, 1e-10)
        refs.append((w.values(), x.cpu().numpy(), its))
    torch.cuda.synchronize()
    wrong = []

    def loop(i):
        try:
            w, b = works[i], rhs[i]
            for _ in range(10):
                w.assemble()
                x, _, its, _, _ = fb.cg_solve(w.K, None, b, None, 5000, 1e-10)
                values, xr, it = refs[i]
                if not (same(w.values(), values) and np.array_equal(x.cpu().numpy(), xr) and its == it):
                    wrong.append(i)
        except Exception as e:                           # a thread's error would be lost
            wrong.append((i, repr(e)))

    threads = [threading.Thread(target=loop, args=(i,)) for i in range(len(works))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
