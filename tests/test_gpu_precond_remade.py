"""A preconditioner made anew on a kept matrix, as every time step of a program with changing values
does: the solve's captured chunk is the new preconditioner's, whatever address it came to lie at."""
import gc

import numpy as np
import pytest

from gpu_problems import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


@pytest.mark.parametrize("kind", ["ilu0", "ssor"])
def test_made_anew(fb, kind):
    import torch
    pr = build(fb, "helmholtz_sin", 18, 2)
    K, (ip, ix) = pr["K"], pr["P"].to_host()
    rows, values = np.repeat(np.arange(K.nrows), np.diff(ip)), K.data
    b = torch.as_tensor(np.random.default_rng(4).standard_normal(K.nrows)).cuda()
    make = fb.ILU0Preconditioner if kind == "ilu0" else (lambda M: fb.SSORPreconditioner(M, 1.3))
    for step in range(8):
        d = np.exp(np.random.default_rng(step).uniform(-2.0, 2.0, K.nrows))
        scaled = d[rows] * values * d[ix]
        K.set_data(scaled)
        M = make(K)
        x, conv, its, _, _ = fb.cg_solve(K, M, b, None, 5000, 1e-10)
        other = fb.CSRMatrix.from_arrays(K.nrows, K.nrows, ip, ix, scaled)
        N = make(other)
        y, conv2, its2, _, _ = fb.cg_solve(other, N, b, None, 5000, 1e-10)
        assert conv and conv2 and its == its2 and torch.equal(x, y)
        del M, N, other
        gc.collect()
