"""The pattern builder and the scatter map on arbitrary cell -> dof maps (csrc/pattern.cu), bit for bit
against numpy: rows of few candidates (sorted in registers), of more than 8 cells, of more columns
than a thread keeps, without cells, constrained entries, and a map whose rows are not kept between
the passes (past the context's scratch)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fb():
    import femd_b200
    return femd_b200


def device_pattern(fb, n, dofs):
    import torch
    from femd_b200 import _native as N
    ctx = fb.context()
    d = torch.as_tensor(np.ascontiguousarray(dofs, dtype=np.int32)).cuda()
    h = C.c_void_p()
    ctx.enter()
    N.check(fb.lib.femd_cuda_pattern_from_cells(ctx.h, n, dofs.shape[0], dofs.shape[1], C.c_void_p(d.data_ptr()), C.byref(h)))
    P = fb.SparsityPattern(h, ctx)
    P.ncells, P.nloc = dofs.shape
    return P


def numpy_pattern(n, dofs):
    i, j = np.repeat(dofs, dofs.shape[1], axis=1).reshape(-1), np.tile(dofs, (1, dofs.shape[1])).reshape(-1)
    inside = (i >= 0) & (j >= 0)
    keys, inv = np.unique(i[inside].astype(np.int64) * n + j[inside], return_inverse=True)
    ip = np.zeros(n + 1, dtype=np.int64)
    np.add.at(ip, keys // n + 1, 1)
    where = np.full(i.size, -1, dtype=np.int32)
    where[inside] = inv
    return np.cumsum(ip), keys % n, where


def cells(kind, nloc, rng):
    """A cell map without a repeated dof within a cell."""
    if kind == "window":          # neighbours share dofs: few candidates a row
        ncells = 700
        d = (nloc - 1) * np.arange(ncells)[:, None] + np.arange(nloc)
    elif kind == "hub":           # one dof in every cell: a row of all cells and of many columns
        ncells = 1000 // nloc
        d = np.zeros((ncells, nloc), dtype=np.int64)
        d[:, 1:] = 1 + np.arange(ncells * (nloc - 1)).reshape(ncells, nloc - 1)
    else:                         # random: rows of 0 to some 20 cells
        n, ncells = 400, 900
        d = np.stack([rng.choice(n - 5, nloc, replace=False) for _ in range(ncells)])
    n = int(d.max()) + 1 + 5      # five rows without cells
    perm = rng.permutation(n)
    d = perm[np.stack([rng.permutation(row) for row in d])]
    d[rng.random(d.shape) < 0.05] = -1
    return n, d.astype(np.int64)


@pytest.mark.parametrize("kind", ["window", "hub", "random"])
@pytest.mark.parametrize("nloc", [1, 3, 4, 6, 10, 15])
def test_arbitrary_maps(fb, kind, nloc):
    if kind == "hub" and nloc == 1:
        pytest.skip("a hub needs another dof")
    n, d = cells(kind, nloc, np.random.default_rng(nloc))
    P = device_pattern(fb, n, d)
    ip, ix, where = numpy_pattern(n, d)
    gip, gix = P.to_host()
    assert np.array_equal(gip, ip) and np.array_equal(gix, ix)
    assert np.array_equal(fb.scatter_map_2d(P).cpu().numpy(), where)


def test_past_the_scratch(fb):
    """Cells of 10 dofs that share 2 with the next: 68 M candidate columns."""
    ncells, nloc = 680000, 10
    d = 8 * np.arange(ncells)[:, None] + np.arange(nloc)
    n = 8 * ncells + 2
    P = device_pattern(fb, n, d)
    gip, gix = P.to_host()
    first = np.maximum(0, 8 * ((np.arange(n) - 2) // 8))            # the first cell with the dof starts here
    last = np.minimum(n, 8 * np.minimum(np.arange(n) // 8, ncells - 1) + nloc)
    assert np.array_equal(np.diff(gip), last - first)
    start = np.repeat(first - gip[:-1], last - first)
    assert np.array_equal(gix, start + np.arange(gix.size))
