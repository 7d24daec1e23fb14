"""An assembly that a CUDA graph replays keeps the tables it read (weights, reference values, pair tensors)
however many other forms the pattern assembles in between, and takes them along where the form is met
for the first time in the capture."""
import numpy as np
import pytest

from gpu_problems import PI

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


@pytest.mark.parametrize("first_met", [False, True])
@pytest.mark.parametrize("k", [1, 2, 3])
def test_other_forms_between(fb, k, first_met):
    import torch
    V = fb.LagrangeSpace2D(fb.rectangle_mesh(0, 0, 1, 1, 20, 20), k, bc="dirichlet")
    P = V.pattern()
    K, L = fb.CSRMatrix(P), fb.CSRMatrix(P)
    one, sin = fb.Coef.const(1.0), fb.Coef.sinsin(1.0, 0.5, 2 * PI, 3 * PI)
    f = torch.zeros(V.dim, dtype=torch.float64, device="cuda")
    Q = V.cache(2 * k + 1)

    def assemble(K, f):
        fb.assemble_matrix_2d(Q, Q, [1, 2, 0], [1, 2, 0], [one, one, one], K, jacobi=False)
        fb.assemble_matrix_2d(Q, Q, [1, 2], [1, 2], [sin, sin], K, jacobi=False)
        fb.assemble_vector_2d(Q, [0], [sin], P, out=f)

    def others():
        for d in range(2 * k + 2, 2 * k + 9):             # every one another rule, and larger
            R = V.cache(d)
            fb.assemble_matrix_2d(R, R, [1, 2], [1, 2], [one, one], L, jacobi=False)
            fb.assemble_vector_2d(R, [0], [sin], P)

    g = torch.cuda.CUDAGraph()
    if first_met:
        fb.assemble_matrix_2d(V.cache(1), V.cache(1), [1, 2], [1, 2], [one, one], L, jacobi=False)   # the row offsets
    else:
        assemble(K, f)
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=K.ctx.stream, capture_error_mode="thread_local"):
        assemble(K, f)
    M, h = fb.CSRMatrix(P), torch.zeros_like(f)
    assemble(M, h)                                        # not replayed yet: the tables are there all the same
    ref, rf = M.data, h.cpu().numpy()
    for _ in range(3):
        others()
        K.data_tensor().zero_()
        f.zero_()
        torch.cuda.synchronize()
        g.replay()
        torch.cuda.synchronize()
        assert np.array_equal(K.data, ref) and np.array_equal(f.cpu().numpy(), rf)
    E = fb.CSRMatrix(P)
    fb.assemble_matrix_2d(Q, Q, [1, 2], [1, 2], [sin, sin], E, jacobi=False, exact=True)
    assert np.abs(E.data - ref).max() <= 1e-12 * np.abs(ref).max()
