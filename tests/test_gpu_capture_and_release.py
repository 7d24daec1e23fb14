"""Threads with a context each: one releases memory (which waits for the device) while the others capture
their solves' chunks.  Neither gets in the other's way."""
import threading

import numpy as np
import pytest

from gpu_problems import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


def test_release_beside_captures(fb):
    import torch
    pr = build(fb, "helmholtz_sin", 24, 2)
    (ip, ix), data, n = pr["P"].to_host(), pr["K"].data, pr["K"].nrows
    b = np.random.default_rng(0).standard_normal(n)

    def fresh():                                          # on the calling thread's context
        return fb.CSRMatrix.from_arrays(n, n, ip, ix, data)

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
        rhs = [torch.as_tensor(b).cuda() for _ in mats]
        return fb.Batch(mats).solve(rhs, tol=1e-10, mixed=True, engine="lockstep")[0][1]

    solves = [mixed, ilu0, lockstep]
    refs = [s().cpu().numpy() for s in solves]
    wrong, done = [], threading.Event()

    def solving(i):
        try:
            for _ in range(10):
                if not np.array_equal(solves[i]().cpu().numpy(), refs[i]):
                    wrong.append(i)
        except BaseException as e:
            wrong.append((i, repr(e)))

    def releasing():
        try:
            while not done.is_set():
                fresh()
        except BaseException as e:
            wrong.append(("release", repr(e)))

    other = threading.Thread(target=releasing)
    threads = [threading.Thread(target=solving, args=(i,)) for i in range(3)]
    other.start()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    done.set()
    other.join()
    assert not wrong
