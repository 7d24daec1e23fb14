"""An application of ILU(0) or SSOR whose wait for its copies runs out: z is NaN and nothing else is
touched, the solve says so, and the preconditioner works as before afterwards."""
import numpy as np
import pytest

from gpu_problems import build

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


# z in shared memory, z in global memory (P2 100 x 100: 39,601 rows), a level read where it lies (P3)
@pytest.mark.parametrize("N,k", [(16, 2), (100, 2), (40, 3)])
@pytest.mark.parametrize("kind", ["ilu0", "ssor"])
def test_wait_runs_out(fb, kind, N, k):
    import torch
    K = build(fb, "helmholtz_sin", N, k)["K"]
    M = fb.ILU0Preconditioner(K) if kind == "ilu0" else fb.SSORPreconditioner(K, 1.2)
    r = torch.as_tensor(np.random.default_rng(2).standard_normal(K.nrows)).cuda()
    z = M.apply(r)
    assert torch.isfinite(z).all()
    M.debug(spin_limit=0)
    assert torch.isnan(M.apply(r)).all()
    with pytest.raises(RuntimeError, match="waited too long"):
        fb.cg_solve(K, M, r, None, 50, 1e-10)
    # a few polls: the copies are there or they are not, never half of them
    for polls in range(1, 6):
        M.debug(spin_limit=polls)
        for _ in range(3):
            y = M.apply(r)
            assert torch.equal(y, z) or torch.isnan(y).all()
    M.debug()
    assert torch.equal(M.apply(r), z)
    x, conv, its, _, brk = fb.cg_solve(K, M, r, None, 5000, 1e-8)
    assert conv and not brk
