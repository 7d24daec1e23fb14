"""Host threads on one context, whose scratch and status words they share: pattern builds, first
assemblies (with the inverse diagonal) of new patterns and of one that two threads share, and zero
diagonals, which each thread is told of and no other."""
import threading

import numpy as np
import pytest
import scipy.sparse as sp

from gpu_problems import PI

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


def in_threads(jobs):
    """Every job in a thread of its own; what any of them raised."""
    wrong = []

    def call(job):
        try:
            job()
        except BaseException as e:
            wrong.append(repr(e))

    threads = [threading.Thread(target=call, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return wrong


def assembled(fb, ctx, V, P, coef):
    Q = V.cache(2 * V.degree + 1)
    K = fb.CSRMatrix(P)
    fb.assemble_matrix_2d(Q, Q, [1, 2, 0], [1, 2, 0], [fb.Coef.const(1.0), coef, coef], K)
    return K.data, K.inv_tensor().cpu().numpy()


def test_builds_and_first_assemblies(fb):
    ctx = fb.context()
    coef = fb.Coef.sinsin(1.0, 0.5, 2 * PI, 3 * PI)
    spaces = [fb.LagrangeSpace2D(fb.rectangle_mesh(0, 0, 1, 1, N, N), k, bc="dirichlet") for N, k in ((21, 1), (33, 3), (60, 2), (9, 3))]
    for V in spaces:
        V.cell_dofs_device(ctx)
    refs = [assembled(fb, ctx, V, fb.cell_pattern(V, V, ctx), coef) for V in spaces]

    def job(i):
        def run():
            for _ in range(15):
                P = fb.cell_pattern(spaces[i], spaces[i], ctx)
                data, inv = assembled(fb, ctx, spaces[i], P, coef)
                assert np.array_equal(data, refs[i][0]) and np.array_equal(inv, refs[i][1])
        return run

    assert not in_threads([job(i) for i in range(4)])


def test_one_new_pattern_in_two_threads(fb):
    ctx = fb.context()
    coef = fb.Coef.sinsin(1.0, 0.5, 2 * PI, 3 * PI)
    V = fb.LagrangeSpace2D(fb.rectangle_mesh(0, 0, 1, 1, 50, 50), 2, bc="dirichlet")
    V.cell_dofs_device(ctx)
    ref = assembled(fb, ctx, V, fb.cell_pattern(V, V, ctx), coef)
    for _ in range(10):
        P = fb.cell_pattern(V, V, ctx)

        def job():
            data, inv = assembled(fb, ctx, V, P, coef)
            assert np.array_equal(data, ref[0]) and np.array_equal(inv, ref[1])

        assert not in_threads([job, job])


def test_zero_diagonals_are_told_to_their_thread(fb):
    ctx = fb.context()
    n = 400

    def job(bad):
        d = np.ones(n)
        if bad >= 0:
            d[bad] = 0.0
        K = fb.CSRMatrix.from_arrays(n, n, np.arange(n + 1), np.arange(n), d, ctx=ctx)

        def run():
            for _ in range(200):
                if bad < 0:
                    fb.JacobiPreconditioner(K)
                else:
                    with pytest.raises(ValueError, match=f"row {bad}$"):
                        fb.JacobiPreconditioner(K)
        return run

    assert not in_threads([job(b) for b in (3, -1, 77, -1)])


def test_first_solves_beside_assemblies(fb):
    """A solve's first call on a matrix captures its chunk of iterations; what other threads queue on the
    context's stream meanwhile is not part of it."""
    import torch
    ctx = fb.context()
    coef = fb.Coef.sinsin(1.0, 0.5, 2 * PI, 3 * PI)
    V = fb.LagrangeSpace2D(fb.rectangle_mesh(0, 0, 1, 1, 24, 24), 2, bc="dirichlet")
    V.cell_dofs_device(ctx)
    P = fb.cell_pattern(V, V, ctx)
    ip, ix = P.to_host()
    data, inv = assembled(fb, ctx, V, P, coef)
    b = torch.as_tensor(np.random.default_rng(0).standard_normal(V.dim)).cuda()

    def fresh():
        return fb.CSRMatrix.from_arrays(V.dim, V.dim, ip, ix, data, ctx=ctx)

    def mixed():
        K = fresh()
        return fb.cg_solve(K, fb.JacobiPreconditioner(K), b, None, 5000, 1e-10, mixed=True)[0]

    def ilu0():
        K = fresh()
        return fb.cg_solve(K, fb.ILU0Preconditioner(K), b, None, 5000, 1e-10)[0]

    def lockstep():
        mats = [fresh(), fresh()]
        for K in mats:
            fb.JacobiPreconditioner(K)
        return fb.Batch(mats, ctx=ctx).solve([b, b], tol=1e-10, mixed=True, engine="lockstep")[0][1]

    solves = [mixed, ilu0, lockstep]
    refs = [s().cpu().numpy() for s in solves]

    def solving(s, ref):
        def run():
            for _ in range(8):
                assert np.array_equal(s().cpu().numpy(), ref)
        return run

    def assembling():
        for _ in range(60):
            d, i = assembled(fb, ctx, V, P, coef)
            assert np.array_equal(d, data) and np.array_equal(i, inv)

    assert not in_threads([solving(s, r) for s, r in zip(solves, refs)] + [assembling])
