"""Measured cases: what a user of femd_b200 has it do, through its public entry points.

    listed()             the fixed cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program holds before the call: meshes, spaces, matrices, vectors
    run(state)           one pass
    work(case)           the bytes and operations a pass cannot do without
    exact(case, seed)    the pass's result in float64 by plain torch

The kinds of work, by where they stand in a program:

    pattern   a new mesh: the sparsity pattern and the element -> position map
    matrix    a (re)assembly on a kept pattern, with the Jacobi inverse diagonal
    load      a load vector
    cg        a Jacobi-PCG solve, FP64 or with the FP32 inner iteration
    ilu0      CG with ILU(0), the default preconditioner of the "cg" backend
    heat      a backward-Euler step (M + dt K) u' = M u from the previous state
    solve     solve(a, L): two compiled forms assembled, the solver built and run
    batch     many Poisson problems of mixed sizes solved together
"""
import math

import numpy as np
import torch

import femd_b200 as fb
from femd_b200 import workloads
from femd_b200.forms import Form2D, Integrand, SparseSolver, solve

PI = math.pi
# form -> test codes, trial codes, the form whose quadrature degree it takes
FORMS = {"poisson": ([1, 2], [1, 2], "gradgrad"), "helmholtz": ([1, 2, 0], [1, 2, 0], "helmholtz"),
         "mass": ([0], [0], "mass"), "varcoef": ([1, 2], [1, 2], "varcoef")}


def listed():
    return [
        # one step of the reference's heat example (P2, 20 x 20, dt = 1e-3): the smallest solve,
        # taken a hundred times in a row
        dict(name="heat_n20_p2", kind="heat", N=20, k=2, dt=1e-3),
        # solve(a, L) at the small configuration (P3, 32 x 32), with a coefficient of x and y
        dict(name="solve_n32_p3", kind="solve", N=32, k=3),
        # a solve with the default preconditioner of the "cg" backend
        dict(name="ilu0_n64_p2", kind="ilu0", N=64, k=2),
        # one request of the mixed-size stream, plain FP64: the middle and the largest of its range
        dict(name="cg_n137_p2", kind="cg", N=137, k=2, form="poisson", mixed=False),
        dict(name="cg_n216_p3", kind="cg", N=216, k=3, form="poisson", mixed=False),
        # the plain method at scale, FP64: 2.4 M unknowns, a matrix of three times the L2 cache
        dict(name="cg_n768_p2", kind="cg", N=768, k=2, form="helmholtz", mixed=False),
        # the precision configuration: a varying coefficient, 1 M unknowns, FP32 inner iteration
        dict(name="mixed_n512_p2", kind="cg", N=512, k=2, form="varcoef", mixed=True),
        # a slice of the mixed-size stream solved together
        dict(name="batch_12", kind="batch", nprob=12, nmin=16, nmax=256, mix=0),
        # a new mesh of half a million triangles
        dict(name="pattern_n512_p2", kind="pattern", N=512, k=2),
        # the matrix and the load vector of the method at scale; re-assembled as data change
        dict(name="matrix_n1024_p2", kind="matrix", N=1024, k=2, form="helmholtz"),
        dict(name="load_n1024_p2", kind="load", N=1024, k=2, coef="sinsin"),
        # the matrix of the precision configuration
        dict(name="varcoef_n512_p2", kind="matrix", N=512, k=2, form="varcoef"),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One case of the ranges above: mesh sizes spread over their logarithm, degrees 1 to 3."""
    kind = rng.choice(["heat", "solve", "ilu0", "cg", "cg", "cg", "mixed", "batch", "pattern", "matrix", "matrix", "load"])
    k = rng.randint(1, 3)
    if kind == "heat":
        return dict(kind=kind, N=_size(rng, 16, 256), k=rng.randint(1, 2), dt=math.exp(rng.uniform(math.log(1e-4), math.log(1e-1))))
    if kind == "solve":
        return dict(kind=kind, N=_size(rng, 8, 128), k=k)
    if kind == "ilu0":
        return dict(kind=kind, N=_size(rng, 8, 96), k=k)
    if kind == "cg":
        return dict(kind=kind, N=_size(rng, 16, 1024 // k), k=k, form=rng.choice(["poisson", "helmholtz", "varcoef"]), mixed=False)
    if kind == "mixed":
        return dict(kind="cg", N=_size(rng, 32, 1024 // k), k=k, form="varcoef", mixed=True)
    if kind == "batch":
        return dict(kind=kind, nprob=rng.randint(4, 12), nmin=16, nmax=rng.randint(64, 256), mix=rng.randint(1, 1000))
    if kind == "pattern":
        return dict(kind=kind, N=_size(rng, 16, 1024 // k), k=k)
    if kind == "matrix":
        return dict(kind=kind, N=_size(rng, 16, 1536 // k), k=k, form=rng.choice(list(FORMS)))
    return dict(kind=kind, N=_size(rng, 16, 1536 // k), k=k, coef=rng.choice(["sinsin", "field"]))


# ---- the inputs, by plain numpy (shared by prepare and exact) ----------------------------------
def _rng(seed, salt=0):
    return np.random.default_rng([int(seed), salt])


def _grid(N):
    """rectangle_mesh(0, 0, 1, 1, N, N): points and triangles."""
    t = np.arange(N + 1) / N
    pts = np.stack([np.tile(t, N + 1), np.repeat(t, N + 1)], axis=1)
    a = (np.arange(N)[:, None] * (N + 1) + np.arange(N)[None, :]).reshape(-1)
    b, c, d = a + 1, a + N + 2, a + N + 1
    return pts, np.stack([a, b, c, a, c, d], axis=1).reshape(-1, 3)


def _mesh_arrays(case, seed):
    """The case's mesh. The matrix and load cases move the inner vertices (a re-assembly follows
    moved or graded meshes); the pattern cases turn one diagonal in ten, so that vertices have
    four to eight neighbours as a mesh generator's do; the solves run on the regular mesh."""
    N = case["N"]
    pts, tris = _grid(N)
    if case["kind"] in ("matrix", "load"):
        move = _rng(seed, 1).uniform(-0.15 / N, 0.15 / N, pts.shape)
        inner = ((pts > 0) & (pts < 1)).all(axis=1)
        pts[inner] += move[inner]
    if case["kind"] == "pattern":
        q = tris.reshape(-1, 6).copy()
        turn = _rng(seed, 2).random(q.shape[0]) < 0.1
        a, b, c, d = q[:, 0], q[:, 1], q[:, 2], q[:, 5]
        q = np.where(turn[:, None], np.stack([a, b, d, b, c, d], axis=1), q)
        tris = q.reshape(-1, 3)
    return pts, np.ascontiguousarray(tris, dtype=np.int32)


def _params(case, seed):
    """Coefficients of the forms: a constant as the stream draws it, the varying ones near the
    configurations' own."""
    r = _rng(seed, 3)
    return dict(c=float(np.exp(r.uniform(np.log(0.1), np.log(10.0)))), amp=float(r.uniform(0.3, 0.6)), f=float(r.uniform(15.0, 25.0)))


def _dof_vector(n, seed, salt):
    return _rng(seed, salt).standard_normal(n)


def _terms(form, p):
    """(coefficient per term): a number, or (p0, p1, a, b) for p0 + p1 sin(a x) sin(b y)."""
    if form == "varcoef":
        return [(1.0, p["amp"], 2 * PI, 2 * PI)] * 2
    return {"poisson": [p["c"]] * 2, "helmholtz": [p["c"], p["c"], 1.0], "mass": [p["c"]]}[form]


def _batch_spec(case, seed):
    """The mixed-size stream's draws: mesh size and degree uniform (the case's own mix), the
    constant log-uniform."""
    r, sizes = _rng(seed, 5), np.random.default_rng([case["mix"], 6])
    return [dict(N=int(sizes.integers(case["nmin"], case["nmax"] + 1)), k=int(sizes.integers(1, 4)),
                 c=float(np.exp(r.uniform(np.log(0.1), np.log(10.0)))), seed=int(r.integers(1 << 31))) for _ in range(case["nprob"])]


# ---- the product's side ------------------------------------------------------------------------
def _space(case, seed):
    pts, tris = _mesh_arrays(case, seed)
    return fb.LagrangeSpace2D(fb.Mesh2D(pts, tris), case["k"], bc="dirichlet", numbering="device")


def _coefs(terms):
    return [fb.Coef.sinsin(*t) if isinstance(t, tuple) else fb.Coef.const(t) for t in terms]


def _matrix(V, form, terms):
    a, b, deg = FORMS[form]
    Q = V.cache(fb.quad_degree(deg, V.degree))
    K = fb.CSRMatrix(V.pattern())
    fb.assemble_matrix_2d(Q, Q, a, b, _coefs(terms), K)
    return K


def _cuda(a):
    return torch.as_tensor(a).cuda()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        cache = workloads.SpaceCache()
        probs = [workloads.build_poisson(s, cache) for s in _batch_spec(case, seed)]
        for s in cache.spaces.values():
            s["P"].batch_layout()
        return dict(kind=kind, B=fb.Batch([K for K, _ in probs]), b=[b for _, b in probs], cache=cache)
    p = _params(case, seed)
    V = _space(case, seed)
    st = dict(kind=kind, V=V)
    if kind == "pattern":
        return st
    if kind == "matrix":
        a, b, deg = FORMS[case["form"]]
        st.update(Q=V.cache(fb.quad_degree(deg, V.degree)), a=a, b=b, c=_coefs(_terms(case["form"], p)), K=fb.CSRMatrix(V.pattern()))
        return st
    if kind == "load":
        V.pattern()
        if case["coef"] == "sinsin":
            st.update(Q=V.cache(fb.quad_degree("rhs_data", V.degree)), c=[fb.Coef.sinsin(0.0, p["f"], PI, PI)])
        else:
            st.update(Q=V.cache(fb.quad_degree("rhs_field", V.degree)), c=[fb.Coef.field(_cuda(_dof_vector(V.dim, seed, 4)))])
        return st
    if kind == "heat":
        M = _matrix(V, "mass", [1.0])
        A = M.combine(_matrix(V, "poisson", [1.0, 1.0]), 1.0, case["dt"])
        st.update(M=M, A=A, pc=fb.JacobiPreconditioner(A), u=_cuda(_dof_vector(V.dim, seed, 4)))
    elif kind == "solve":
        k = V.degree
        coef = (Integrand.varcoef(), [], [0, 1, 2])
        data = (Integrand.varcoef(), [], [0, 1, 2])
        st.update(a=Form2D.build(V, [(1, 1, coef), (2, 2, coef)], fb.quad_degree("varcoef", k), consts=[1.0, p["amp"], 2 * PI]),
                  L=Form2D.build(V, [(0, data)], fb.quad_degree("rhs_data", k), consts=[0.0, p["f"], PI]))
    elif kind == "ilu0":
        st.update(S=SparseSolver(_matrix(V, "poisson", [p["c"], p["c"]]), "cg", tol=1e-12), b=_cuda(_dof_vector(V.dim, seed, 4)))
    else:
        A = _matrix(V, case["form"], _terms(case["form"], p))
        st.update(A=A, pc=fb.JacobiPreconditioner(A), b=_cuda(_dof_vector(V.dim, seed, 4)), mixed=case["mixed"])
    return st


def _view(t, owner):
    """A view of device memory that a handle owns: the handle lives as long as the view."""
    t.owner = owner
    return t


def run(st):
    kind = st["kind"]
    if kind == "pattern":
        P = fb.cell_pattern(st["V"], st["V"])
        return _view(fb.scatter_map_2d(P), P)
    if kind == "matrix":
        K = fb.assemble_matrix_2d(st["Q"], st["Q"], st["a"], st["b"], st["c"], st["K"])
        return _view(K.data_tensor(), K), _view(K.inv_tensor(), K)
    if kind == "load":
        return fb.assemble_vector_2d(st["Q"], [0], st["c"])
    if kind == "heat":
        b = st["M"].matvec(st["u"])
        return b, fb.cg_solve(st["A"], st["pc"], b, st["u"], 100000, 1e-10)[0]
    if kind == "solve":
        return solve(st["a"], st["L"], tol=1e-10)
    if kind == "ilu0":
        return st["S"].solve(st["b"])
    # 1e-12, the tighter of the tolerances in use: the solve's own error then is well below what
    # the results are compared to
    if kind == "batch":
        return st["B"].solve(st["b"], tol=1e-12, mixed=True, engine="lockstep")[0]
    return fb.cg_solve(st["A"], st["pc"], st["b"], None, 100000, 1e-12, mixed=st["mixed"])[0]


# ---- what a pass cannot do without -------------------------------------------------------------
def _counts(N, k):
    """(unknowns, nonzeros, cells, vertices) of P_k on the N x N mesh, its boundary eliminated."""
    m = k * N - 1
    row = {1: 7.0, 2: 11.5, 3: 16.5}[k]
    return m * m, row * m * m, 2 * N * N, (N + 1) ** 2


def _iterations(N, k, digits):
    return 0.42 * k * N * digits


def _solve_work(n, nnz, its):
    """The matrix, its inverse diagonal and the vectors once; an SpMV, two dot products and three
    vector updates an iteration."""
    return 12.0 * nnz + 4.0 * n + 24.0 * n, its * (2.0 * nnz + 13.0 * n)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        mid = 0.5 * (case["nmin"] + case["nmax"])
        one = [_solve_work(*_counts(mid, k)[:2], _iterations(mid, k, 12)) for k in (1, 2, 3)]
        return {"bytes": case["nprob"] * sum(w[0] for w in one) / 3, "flops": case["nprob"] * sum(w[1] for w in one) / 3}
    N, k = case["N"], case["k"]
    n, nnz, cells, verts = _counts(N, k)
    nloc = (k + 1) * (k + 2) // 2
    geometry = 16.0 * verts + 12.0 * cells
    if kind == "pattern":
        return {"bytes": 4.0 * cells * nloc + 4.0 * (n + nnz) + 4.0 * cells * nloc * nloc, "flops": 0}
    if kind == "matrix":
        # the pattern's columns stand for the positions; the values and the inverse diagonal are written
        terms = 4 if case["form"] == "helmholtz" else 3
        return {"bytes": geometry + 4.0 * cells * nloc + 4.0 * nnz + 8.0 * nnz + 8.0 * n, "flops": 2.0 * terms * cells * nloc * nloc}
    if kind == "load":
        field = 8.0 * n if case["coef"] == "field" else 0.0
        return {"bytes": geometry + 4.0 * cells * nloc + 8.0 * n + field, "flops": 2.0 * 7 * cells * nloc}
    if kind == "heat":
        its = min(_iterations(N, k, 10), 20 + 2.0 * k * N * math.sqrt(case["dt"]) * 10)
        b, f = _solve_work(n, nnz, its)
        return {"bytes": b + 12.0 * nnz + 12.0 * n, "flops": f + 2.0 * nnz}
    if kind == "solve":
        b, f = _solve_work(n, nnz, _iterations(N, k, 10))
        return {"bytes": b + geometry + 8.0 * cells * nloc + 8.0 * nnz, "flops": f}
    b, f = _solve_work(n, nnz, _iterations(N, k, 12) / (3.0 if kind == "ilu0" else 1.0))
    return {"bytes": b, "flops": f * (2.0 if kind == "ilu0" else 1.0)}


# ---- the results by plain torch in float64 -----------------------------------------------------
def _numbering(tris, nverts, k):
    """Dofs of each cell (-1 on the boundary) and their count: vertices, then the k - 1 nodes of
    each edge (edges in the order of their first appearance, edge i of a cell from its local
    vertex i + 1 to i + 2, nodes from the smaller vertex on), then the inner nodes."""
    nc, de, ni = tris.shape[0], k - 1, (k - 1) * (k - 2) // 2
    a, b = tris[:, [1, 2, 0]], tris[:, [2, 0, 1]]
    key = (torch.minimum(a, b) * nverts + torch.maximum(a, b)).reshape(-1)
    uniq, inv, count = torch.unique(key, return_inverse=True, return_counts=True)
    first = torch.full((uniq.numel(),), key.numel(), device=tris.device).scatter_reduce_(0, inv, torch.arange(key.numel(), device=tris.device), "amin")
    rank = torch.empty_like(first)
    rank[torch.argsort(first)] = torch.arange(uniq.numel(), device=tris.device)
    edge = rank[inv].reshape(nc, 3)
    j = torch.arange(de, device=tris.device)
    at = torch.where((a > b)[:, :, None], de - 1 - j, j)
    nodes = [tris, (nverts + edge[:, :, None] * de + at).reshape(nc, 3 * de),
             nverts + uniq.numel() * de + torch.arange(nc * ni, device=tris.device).reshape(nc, ni)]
    raw = torch.cat(nodes, dim=1)
    keep = torch.ones(nverts + uniq.numel() * de + nc * ni, dtype=torch.bool, device=tris.device)
    outer = (count == 1)[inv].reshape(nc, 3)
    keep[a[outer]] = False
    keep[b[outer]] = False
    keep[nodes[1].reshape(nc, 3, de)[outer].reshape(-1)] = False
    new = torch.where(keep, torch.cumsum(keep, 0) - 1, -1)
    return new[raw], int(keep.sum())


def _nodes(k):
    """Reference coordinates of the local nodes, in the numbering's order."""
    v = np.array([[0.0, 0.0], [1.0, 0.0], [0.0, 1.0]])
    pts = list(v)
    for i in range(3):
        s, e = v[(i + 1) % 3], v[(i + 2) % 3]
        pts += [s + (e - s) * j / k for j in range(1, k)]
    pts += [np.array([i, j]) / k for j in range(1, k) for i in range(1, k - j)]
    return np.array(pts)


def _basis(k, xi, eta):
    """Values and both derivatives of the Lagrange basis at points: (3, points, nodes)."""
    powers = [(i, j) for i in range(k + 1) for j in range(k + 1 - i)]

    def table(x, y, dx, dy):
        c = []
        for i, j in powers:
            u = i * x ** max(i - 1, 0) if dx else x ** i
            v = j * y ** max(j - 1, 0) if dy else y ** j
            c.append(u * v)
        return np.stack(c, axis=1)

    n = _nodes(k)
    inv = np.linalg.inv(table(n[:, 0], n[:, 1], 0, 0))
    return np.stack([table(xi, eta, *d) @ inv for d in ((0, 0), (1, 0), (0, 1))])


def _degree(form, k):
    """The quadrature degree of a form: the arguments' degrees, k + 1 for a coefficient of x and y."""
    return max({"poisson": 2 * k - 2, "helmholtz": 2 * k, "mass": 2 * k, "varcoef": 3 * k - 1, "sinsin": 2 * k + 1, "field": 2 * k}[form], 1)


def _rule(degree):
    """The triangle rule of a degree: 1, 3 or 7 points up to degree 5, then Gauss products."""
    if degree <= 1:
        return np.array([1 / 3]), np.array([1 / 3]), np.array([0.5])
    if degree == 2:
        return np.array([1 / 6, 2 / 3, 1 / 6]), np.array([1 / 6, 1 / 6, 2 / 3]), np.full(3, 1 / 6)
    if degree <= 5:
        s = math.sqrt(15.0)
        a, b, wa, wb = (6 - s) / 21, (6 + s) / 21, (155 - s) / 2400, (155 + s) / 2400
        return (np.array([1 / 3, a, 1 - 2 * a, a, b, 1 - 2 * b, b]), np.array([1 / 3, a, a, 1 - 2 * a, b, b, 1 - 2 * b]),
                np.array([9 / 80, wa, wa, wa, wb, wb, wb]))
    gu, wu = np.polynomial.legendre.leggauss((degree + 2) // 2)
    gv, wv = np.polynomial.legendre.leggauss((degree + 3) // 2)
    u, v = np.meshgrid(0.5 * (gu + 1), 0.5 * (gv + 1))
    w = 0.25 * np.outer(wv, wu) * (1 - v)
    return (u * (1 - v)).reshape(-1), v.reshape(-1), w.reshape(-1)


class _Elements:
    """The mesh, numbering and pattern of a case in plain torch."""

    def __init__(self, case, seed):
        pts, tris = _mesh_arrays(case, seed)
        self.k = case["k"]
        self.pts, self.tris = _cuda(pts), _cuda(tris.astype(np.int64))
        self.dofs, self.n = _numbering(self.tris, pts.shape[0], self.k)

    def pattern(self):
        """Row starts, columns, and every element entry's position (-1 at the boundary)."""
        i, j = self.dofs[:, :, None], self.dofs[:, None, :]
        inside = (i >= 0) & (j >= 0)
        key = (i * self.n + j)[inside]
        uniq, inv = torch.unique(key, return_inverse=True)
        self.inside, self.at, self.col = inside, inv, uniq % self.n
        self.row = torch.zeros(self.n + 1, dtype=torch.int64, device=key.device)
        self.row[1:] = torch.cumsum(torch.bincount(uniq // self.n, minlength=self.n), 0)
        where = torch.full(inside.shape, -1, dtype=torch.int32, device=key.device)
        where[inside] = inv.to(torch.int32)
        return where

    def _points(self, degree, lo, hi):
        """Weights x |det J|, basis rows by derivative code, and the physical points of cells lo..hi."""
        xi, eta, w = _rule(degree)
        R = _cuda(_basis(self.k, xi, eta))
        P = self.pts[self.tris[lo:hi]]
        J = torch.stack([P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]], dim=2)
        det = J[:, 0, 0] * J[:, 1, 1] - J[:, 0, 1] * J[:, 1, 0]
        G = torch.linalg.inv(J)                        # d(xi, eta) / d(x, y)
        rows = [R[0].expand(hi - lo, -1, -1)] + [G[:, 0, d, None, None] * R[1] + G[:, 1, d, None, None] * R[2] for d in (0, 1)]
        xy = P[:, 0, :, None] + J @ _cuda(np.stack([xi, eta]))
        return det.abs()[:, None] * _cuda(w), rows, R[0], xy

    def _coef(self, t, xy, values, dofs):
        if isinstance(t, tuple):
            return t[0] + t[1] * torch.sin(t[2] * xy[:, 0]) * torch.sin(t[3] * xy[:, 1])
        if isinstance(t, torch.Tensor):
            return torch.where(dofs >= 0, t[dofs.clamp(min=0)], 0.0) @ values.T
        return torch.full_like(xy[:, 0], t)

    def _chunks(self):
        step = 1 << 17
        return [(lo, min(lo + step, self.tris.shape[0])) for lo in range(0, self.tris.shape[0], step)]

    def matrix(self, form, terms):
        """The values on the pattern."""
        a, b, _ = FORMS[form]
        self.pattern()
        Ke = []
        for lo, hi in self._chunks():
            w, rows, R0, xy = self._points(_degree(form, self.k), lo, hi)
            Ke.append(sum(torch.einsum("eq,eqi,eqj->eij", w * self._coef(c, xy, R0, self.dofs[lo:hi]), rows[s], rows[t])
                          for s, t, c in zip(a, b, terms)))
        Ke = torch.cat(Ke)
        return torch.zeros(self.col.numel(), dtype=torch.float64, device=Ke.device).index_add_(0, self.at, Ke[self.inside])

    def load(self, kind, coef):
        f = torch.zeros(self.n, dtype=torch.float64, device=self.pts.device)
        for lo, hi in self._chunks():
            w, rows, R0, xy = self._points(_degree(kind, self.k), lo, hi)
            d = self.dofs[lo:hi]
            f.index_add_(0, d[d >= 0], (w * self._coef(coef, xy, R0, d) @ R0)[d >= 0])
        return f

    def inverse_diagonal(self, data):
        at = torch.repeat_interleave(torch.arange(self.n, device=data.device), self.row[1:] - self.row[:-1])
        return 1.0 / data[at == self.col]

    def csr(self, data):
        return torch.sparse_csr_tensor(self.row, self.col, data, (self.n, self.n))

    def solve(self, data, b):
        """A x = b by conjugate gradients in torch, down to rounding."""
        A, inv = self.csr(data), self.inverse_diagonal(data)
        x, r = torch.zeros_like(b), b.clone()
        p = inv * r
        rz = torch.dot(r, p)
        stop = 1e-15 * torch.linalg.vector_norm(b)
        for it in range(40000):
            q = A @ p
            alpha = rz / torch.dot(p, q)
            x += alpha * p
            r -= alpha * q
            if it % 50 == 0 and torch.linalg.vector_norm(r) <= stop:
                break
            z = inv * r
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
        return x


def exact(case, seed):
    kind, p = case["kind"], _params(case, seed)
    if kind == "batch":
        out = []
        for s in _batch_spec(case, seed):
            E = _Elements(dict(kind="cg", N=s["N"], k=s["k"]), 0)
            data = E.matrix("poisson", [s["c"]] * 2)
            out.append(E.solve(data, _cuda(np.random.default_rng(s["seed"]).standard_normal(E.n))))
        return out
    E = _Elements(case, seed)
    if kind == "pattern":
        return E.pattern().reshape(-1)
    if kind == "matrix":
        data = E.matrix(case["form"], _terms(case["form"], p))
        return data, E.inverse_diagonal(data)
    if kind == "load":
        if case["coef"] == "sinsin":
            return E.load("sinsin", (0.0, p["f"], PI, PI))
        return E.load("field", _cuda(_dof_vector(E.n, seed, 4)))
    if kind == "heat":
        u = _cuda(_dof_vector(E.n, seed, 4))
        M = E.matrix("mass", [1.0])
        b = E.csr(M) @ u
        return b, E.solve(M + case["dt"] * E.matrix("poisson", [1.0, 1.0]), b)
    if kind == "solve":
        data = E.matrix("varcoef", [(1.0, p["amp"], 2 * PI, 2 * PI)] * 2)
        return E.solve(data, E.load("sinsin", (0.0, p["f"], PI, PI)))
    form = "poisson" if kind == "ilu0" else case["form"]
    return E.solve(E.matrix(form, _terms(form, p)), _cuda(_dof_vector(E.n, seed, 4)))
