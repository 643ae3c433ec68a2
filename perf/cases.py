"""Workloads of the matrix-free path: what is timed, on which inputs, and the 64-bit result.

A case is a dict of plain values.  ``prepare`` builds what a program holds before the call
(1D rules, operator or preconditioner, device vectors) from a seed, ``run`` is one call
through the public entry points, ``work`` the bytes and operations that call cannot do
without, ``exact`` its result in FP64 with plain torch / numpy on the same inputs.

Kinds: "matvec" (``MFOperator.apply``), "fd" (``SingleFD.apply``), "fd_tc" (the BF16
tensor-core apply), "sptime" (space-time ``SingleFD.apply``), "geometry"
(``precompute_coefficients``), "solve" (``EllipticPatchSolver.solve_fp64``) and "batch"
(``BatchedFGMRES`` over several patches).  ``ne1``, ``ne2``, ``ne3``: elements per direction
(absent directions 0), ``p``: degree, ``rule``: "wq2" (weighted quadrature, type 2) or
"gauss" (Gauss-Legendre).
"""
import math

import numpy as np
import torch

from igaops_b200 import GeometryOps, MFOperator, StandardGauss, WeightedQuadrature
from igaops_b200 import precompute_coefficients
from igaops_b200.batch import BatchedFGMRES, PatchBatch
from igaops_b200.fastdiag import SingleFD
from igaops_b200.refine import EllipticPatchSolver

DTYPES = {"f64": torch.float64, "f32": torch.float32}
# elements and degrees of the patches of a "batch" case, relative to its ne1
BATCH_PATCHES = ((2, 1.0), (3, 0.75), (4, 0.5), (3, 1.25), (2, 0.6), (4, 0.8))


def listed():
    return [
        # the operator pair of the library's benchmark: one stiffness and one mass
        # product on a large 3D patch, launch shape tuned once as the README shows
        dict(name="stiffness_3d_p3_128_f64", kind="matvec", op="gradu_gradv", p=3, ne1=128,
             ne2=128, ne3=128, rule="wq2", dtype="f64", tuned=True, st=False, cols=1),
        dict(name="mass_3d_p3_128_f64", kind="matvec", op="u_v", p=3, ne1=128, ne2=128, ne3=128,
             rule="wq2", dtype="f64", tuned=True, st=False, cols=1),
        # the single-precision product of the mixed solvers' inner iterations, on a
        # medium patch of odd size
        dict(name="stiffness_3d_p4_61_f32", kind="matvec", op="gradu_gradv", p=4, ne1=61, ne2=57,
             ne3=63, rule="wq2", dtype="f32", tuned=False, st=False, cols=1),
        # advection term of a convection-diffusion operator
        dict(name="advection_3d_p2_40_f64", kind="matvec", op="gradu_v", p=2, ne1=40, ne2=40,
             ne3=40, rule="wq2", dtype="f64", tuned=False, st=False, cols=1),
        # smallest product: a 2D patch whose Krylov iterations are launch-bound
        dict(name="stiffness_2d_p3_64_f64", kind="matvec", op="gradu_gradv", p=3, ne1=64, ne2=64,
             ne3=0, rule="wq2", dtype="f64", tuned=False, st=False, cols=1),
        # large 2D patch of high degree and odd size
        dict(name="stiffness_2d_p5_301_f64", kind="matvec", op="gradu_gradv", p=5, ne1=301,
             ne2=283, ne3=0, rule="wq2", dtype="f64", tuned=False, st=False, cols=1),
        # preconditioner of the FP64 solves, on the mixed-solve benchmark's patch
        dict(name="fd_3d_p3_96_f64", kind="fd", p=3, ne1=96, ne2=96, ne3=96, dtype="f64"),
        # preconditioner of the mixed-precision solves on the same patch
        dict(name="fd_tc_3d_p3_96", kind="fd_tc", p=3, ne1=96, ne2=96, ne3=96, dtype="f64"),
        # preconditioner of a space-time heat solve (2D in space), serving size
        dict(name="sptime_fd_p3_24_f64", kind="sptime", p=3, ne1=24, ne2=24, ne3=24,
             dtype="f64"),
        # coefficients of a new geometry: paid once per patch before its first product
        dict(name="geometry_3d_p3_64", kind="geometry", p=3, ne1=64, ne2=64, ne3=64),
        # whole FD-preconditioned GMRES solve of one small patch in FP64
        dict(name="solve_fp64_3d_p2_24", kind="solve", p=2, ne1=24, ne2=24, ne3=24),
        # whole mixed-precision solve of several patches at once
        dict(name="solve_batch_3d_40", kind="batch", ne1=40),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec"] * 10 + ["fd"] * 4 + ["fd_tc", "sptime", "sptime", "geometry",
                                                      "solve", "batch"])
    p = rng.choice([2, 3, 4, 5])
    if kind == "matvec":
        two = rng.random() < 0.3
        st = not two and rng.random() < 0.15
        rule = "gauss" if rng.random() < 0.2 else "wq2"
        op = rng.choice(["u_v", "gradu_gradv"] if st else
                        ["u_v", "gradu_gradv", "gradu_gradv", "gradu_v", "u_gradv"])
        if two:
            base = _log(rng, 8, 128 if rule == "gauss" else 320)
        elif st:
            base = _log(rng, 8, 32)
        else:
            base = _log(rng, 8, 36 if rule == "gauss" else 104 if p <= 3 else 88)
        ne = [max(6, int(base * rng.uniform(0.75, 1.2))) for _ in range(2 if two else 3)] + [0]
        return dict(kind=kind, op=op, p=p, ne1=ne[0], ne2=ne[1], ne3=ne[2], rule=rule,
                    dtype=rng.choice(["f64", "f64", "f32"]), tuned=False, st=st,
                    cols=3 if rng.random() < 0.1 and base <= 48 else 1)
    if kind == "fd":
        two = rng.random() < 0.3
        base = _log(rng, 8, 200 if two else 100)
        ne = [max(6, int(base * rng.uniform(0.75, 1.2))) for _ in range(2 if two else 3)] + [0]
        return dict(kind=kind, p=p, ne1=ne[0], ne2=ne[1], ne3=ne[2],
                    dtype=rng.choice(["f64", "f64", "f32"]))
    if kind == "sptime":
        ne = [rng.randint(8, 26) for _ in range(3)]
        return dict(kind=kind, p=p, ne1=ne[0], ne2=ne[1], ne3=ne[2], dtype="f64")
    base = _log(rng, 8, {"fd_tc": 104, "geometry": 64, "solve": 32, "batch": 40}[kind])
    if kind == "batch":
        return dict(kind=kind, ne1=max(12, base))
    ne = [max(6, int(base * rng.uniform(0.75, 1.2))) for _ in range(3)]
    out = dict(kind=kind, p=p, ne1=ne[0], ne2=ne[1], ne3=ne[2])
    return dict(out, dtype=rng.choice(["f64", "f32"])) if kind == "fd_tc" else out


# ------------------------------------------------------------------ inputs
def _elements(case):
    return [case[k] for k in ("ne1", "ne2", "ne3") if case[k]]


def _knots(p, ne):
    return GeometryOps.make_open_knotvector(p, ne)


def _rules(p, elements, rule="wq2"):
    made = {}
    for ne in elements:
        if ne not in made:
            kv = _knots(p, ne)
            made[ne] = (StandardGauss(p, kv, "legendre") if rule == "gauss"
                        else WeightedQuadrature(p, kv, "2"))
    return [made[ne] for ne in elements]


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _coefficients(rules, op, spd, seed, dtype):
    """Smooth coefficient fields over the quadrature points (first direction fastest): a
    symmetric positive definite tensor near the identity, a density near 1, or a velocity."""
    rs = np.random.RandomState(seed)
    grids = [torch.linspace(0.0, 1.0, int(q.nbquadpts), dtype=torch.float64, device="cuda")
             for q in rules]

    def wave(amplitude):
        out = torch.full([1], float(amplitude * rs.uniform(0.5, 1.0)), dtype=torch.float64,
                         device="cuda")
        for g in grids[::-1]:
            out = out.reshape(-1, 1) * torch.sin(
                2 * math.pi * (g * rs.randint(1, 3) + rs.uniform()))[None, :]
        return out.reshape(-1)

    if op == "u_v":
        return (1.0 + wave(0.3)).to(dtype)
    if op == "gradu_gradv":
        c = torch.empty((spd, spd, math.prod(int(q.nbquadpts) for q in rules)), dtype=dtype,
                        device="cuda")
        for i in range(spd):
            c[i, i] = 1.0 + wave(0.2)
            for j in range(i):
                c[i, j] = wave(0.1)
                c[j, i] = c[i, j]
        return c
    return torch.stack([0.5 + wave(0.5) for _ in range(spd)]).to(dtype)


def _vector(n, seed, dtype, cols=1):
    shape = (n,) if cols == 1 else (n, cols)
    return torch.randn(shape, generator=_generator(seed), dtype=torch.float64,
                       device="cuda").to(dtype)


def _ctrlpts(p, elements, seed):
    """Control net of a perturbed unit cube: Greville points displaced by a fraction of the
    element size (the displacement's phase and amplitude depend on the seed)."""
    rs = np.random.RandomState(seed)
    g = []
    for ne in elements:
        kv = _knots(p, ne)
        g.append(np.array([kv[i + 1:i + p + 1].mean() for i in range(len(kv) - p - 1)]))
    grids = [a.reshape(-1) for a in np.meshgrid(*g[::-1], indexing="ij")[::-1]]
    h = 1.0 / max(elements)
    out = []
    for c in grids:
        bump = rs.uniform(0.05, 0.15) * h
        for d in grids:
            bump = bump * np.sin(2 * np.pi * (d + rs.uniform()))
        out.append(c + bump)
    return torch.from_numpy(np.stack(out)).cuda()


def _sizes(rules):
    return (math.prod(int(q.nbctrlpts) for q in rules), math.prod(int(q.nbquadpts) for q in rules))


def _batch_layout(case):
    return [(p, max(6, int(case["ne1"] * f))) for p, f in BATCH_PATCHES]


def _dirichlet(ndim):
    return np.ones((1, ndim, 2), dtype=bool)


# ----------------------------------------------------------- prepare / run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        patches, parts = [], []
        for i, (p, ne) in enumerate(_batch_layout(case)):
            rules = _rules(p, [ne] * 3)
            coefs = _coefficients(rules, "gradu_gradv", 3, seed + i, torch.float64)
            patches.append(PatchBatch.make_patch(rules, coefs, _dirichlet(3)))
            parts.append(_vector(_sizes(rules)[0], seed + i, torch.float64))
        batch = PatchBatch(patches)
        solver = BatchedFGMRES(batch, tolerance=1e-10, restart=12)
        return dict(case=case, solver=solver, b=torch.cat(parts))
    p, elements = case["p"], _elements(case)
    ndim = len(elements)
    dtype = DTYPES[case.get("dtype", "f64")]
    if kind == "geometry":
        return dict(case=case, rules=_rules(p, elements), ctrlpts=_ctrlpts(p, elements, seed))
    rules = _rules(p, elements, case.get("rule", "wq2"))
    n = _sizes(rules)[0]
    if kind == "matvec":
        spd = ndim - 1 if case["st"] else ndim
        coefs = _coefficients(rules, case["op"], spd, seed, dtype)
        ders = None if not case["st"] else ((0, 1) if case["op"] == "u_v" else (0, 0))
        oper = MFOperator(rules, coefs, case["op"], ders, dtype=dtype,
                          nseg="auto" if case["tuned"] else None)
        return dict(case=case, oper=oper, x=_vector(n, seed, dtype, case["cols"]))
    if kind == "solve":
        coefs = _coefficients(rules, "gradu_gradv", 3, seed, torch.float64)
        return dict(case=case, solver=EllipticPatchSolver(rules, coefs, _dirichlet(3)),
                    b=_vector(n, seed, torch.float64))
    if kind == "sptime":
        fd = SingleFD("spacetime")
        fd.compute_space_eigendecomposition(rules[:-1], _dirichlet(ndim - 1))
        fd.compute_time_schurdecomposition(rules[-1])
        fd.update_space_eigenvalues([0.0, 1.0])
    else:
        fd = SingleFD("spatial")
        fd.compute_space_eigendecomposition(rules, _dirichlet(ndim))
        fd.update_space_eigenvalues([0.0, 1.0])
    x = _vector(n, seed, dtype)
    return dict(case=case, fd=fd, x=x, y=torch.empty_like(x))


def run(state):
    kind = state["case"]["kind"]
    if kind == "matvec":
        return state["oper"].apply(state["x"])
    if kind in ("fd", "sptime"):
        return state["fd"].apply(state["x"])
    if kind == "fd_tc":
        state["fd"].space_preconditioner.apply_device_tc(state["x"], state["y"])
        return state["y"]
    if kind == "geometry":
        return precompute_coefficients(state["rules"], state["ctrlpts"])
    if kind == "solve":
        return state["solver"].solve_fp64(state["b"]).solution
    return state["solver"].solve(state["b"]).solution


# -------------------------------------------------------------------- work
def _points(p, ne, rule="wq2"):
    # the type-2 rule has three points per element and p - 1 more at each end
    return ne * (p + 1) if rule == "gauss" else 3 * ne + 2 * p - 1


def _matvec_work(op, p, n, nq, size, spd, cols=1):
    streams = {"u_v": 1, "gradu_gradv": spd * (spd + 1) // 2}.get(op, spd)
    trial = spd if op in ("gradu_gradv", "u_gradv") else 1
    test = spd if op in ("gradu_gradv", "gradu_v") else 1
    points = math.prod(nq)
    flops = 2 * points * ((trial + test) * (p + 1) + trial * test)
    return points * streams * size + 2 * math.prod(n) * size * cols, flops * cols


def _fd_flops(m):
    return 4 * math.prod(m) * sum(m)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        nbytes = flops = 0
        for p, ne in _batch_layout(case):
            n, nq = [ne + p] * 3, [_points(p, ne)] * 3
            b, f = _matvec_work("gradu_gradv", p, n, nq, 8, 3)
            nbytes += b
            flops += f + _fd_flops([v - 2 for v in n])
        return {"bytes": nbytes, "flops": flops}
    p, elements = case["p"], _elements(case)
    n = [ne + p for ne in elements]
    total = math.prod(n)
    size = 8 if case.get("dtype", "f64") == "f64" else 4
    if kind == "geometry":
        points = math.prod(_points(p, ne) for ne in elements)
        return {"bytes": 8 * (10 * points + 3 * total), "flops": points * (18 * (p + 1) + 90)}
    if kind in ("fd", "fd_tc"):
        m = [v - 2 for v in n]
        return {"bytes": 2 * size * total, "flops": _fd_flops(m)}
    if kind == "sptime":
        m = [v - 2 for v in n[:-1]] + [n[-1] - 1]
        mm = math.prod(m)
        return {"bytes": 2 * size * total, "flops": 4 * mm * (sum(m) + m[-1]) + 60 * mm}
    rule = case.get("rule", "wq2")
    nq = [_points(p, ne, rule) for ne in elements]
    if kind == "solve":
        b, f = _matvec_work("gradu_gradv", p, n, nq, 8, 3)
        return {"bytes": b, "flops": f + _fd_flops([v - 2 for v in n])}
    spd = len(n) - 1 if case["st"] else len(n)
    b, f = _matvec_work(case["op"], p, n, nq, size, spd, case["cols"])
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------- exact
def _kron(mats, x):
    """(M_d x ... x M_1) x, first direction fastest."""
    t = x.reshape([m.shape[1] for m in mats[::-1]])
    for k, m in enumerate(mats[::-1]):
        t = torch.movedim(torch.tensordot(m, t, dims=([1], [k])), 0, k)
    return t.reshape(-1)


def _dense(a):
    return torch.from_numpy(np.ascontiguousarray(a.toarray(), dtype=np.float64)).cuda()


def _dense_rules(rules):
    B = [[_dense(q.basis[k]) for k in range(2)] for q in rules]
    W = [[_dense(q.weights[k]) for k in range(4)] for q in rules]
    return B, W


def _product(B, W, coefs, op, spd, st, x):
    """y = sum_ij W(alpha_i) [ C_ij * B(beta_j) x ] with dense 1D factors."""
    ndim = len(B)

    def unit(k):
        return [int(d == k) for d in range(ndim)]

    trial = [unit(j) for j in range(spd)] if op in ("gradu_gradv", "u_gradv") else [[0] * ndim]
    test = [unit(i) for i in range(spd)] if op in ("gradu_gradv", "gradu_v") else [[0] * ndim]
    if st and op == "u_v":
        trial[0][-1] = 1
    y = 0
    for j, b in enumerate(trial):
        u = _kron([B[d][b[d]] for d in range(ndim)], x)
        for i, a in enumerate(test):
            c = (coefs if op == "u_v" else coefs[i, j] if op == "gradu_gradv"
                 else coefs[i] if op == "gradu_v" else coefs[j])
            # a space-time mass term takes the plain test weights in time
            z = [0] * ndim if op == "u_v" else [b[d] + 2 * a[d] for d in range(ndim)]
            y = y + _kron([W[d][z[d]] for d in range(ndim)], c.double() * u)
    return y


def _bspline(p, kv, x):
    """Values and first derivatives of the B-splines at x: (points, functions) each."""
    def table(deg):
        if deg == 0:
            last = np.nonzero(kv[:-1] < kv[1:])[0][-1]
            spans = np.arange(len(kv) - 1)
            at = np.clip(np.searchsorted(kv, x, side="right") - 1, 0, last)
            return (spans[None, :] == at[:, None]).astype(np.float64)
        low = table(deg - 1)
        out = np.zeros((len(x), len(kv) - deg - 1))
        for i in range(out.shape[1]):
            if kv[i + deg] > kv[i]:
                out[:, i] += (x - kv[i]) / (kv[i + deg] - kv[i]) * low[:, i]
            if kv[i + deg + 1] > kv[i + 1]:
                out[:, i] += (kv[i + deg + 1] - x) / (kv[i + deg + 1] - kv[i + 1]) * low[:, i + 1]
        return out

    low = table(p - 1)
    ders = np.zeros((len(x), len(kv) - p - 1))
    for i in range(ders.shape[1]):
        if kv[i + p] > kv[i]:
            ders[:, i] += p / (kv[i + p] - kv[i]) * low[:, i]
        if kv[i + p + 1] > kv[i + 1]:
            ders[:, i] -= p / (kv[i + p + 1] - kv[i + 1]) * low[:, i + 1]
    return table(p), ders


def _pencil(p, ne):
    """1D mass, stiffness and advection matrices by Gauss quadrature."""
    kv = np.concatenate([np.zeros(p), np.linspace(0.0, 1.0, ne + 1), np.ones(p)])
    t, w = np.polynomial.legendre.leggauss(p + 1)
    edges = np.linspace(0.0, 1.0, ne + 1)
    x = np.concatenate([0.5 * (b - a) * t + 0.5 * (a + b) for a, b in zip(edges, edges[1:])])
    ww = np.concatenate([0.5 * (b - a) * w for a, b in zip(edges, edges[1:])])
    N, dN = _bspline(p, kv, x)
    return [torch.from_numpy(a).cuda() for a in (N.T @ (ww[:, None] * N),
                                                 dN.T @ (ww[:, None] * dN),
                                                 N.T @ (ww[:, None] * dN))]


def _eigenpairs(p, ne):
    """Generalized eigenpairs of (stiffness, mass) without the first and last function."""
    M, K, _ = _pencil(p, ne)
    M, K = M[1:-1, 1:-1], K[1:-1, 1:-1]
    L = torch.linalg.cholesky(M)
    C = torch.linalg.solve_triangular(L, K, upper=False)
    C = torch.linalg.solve_triangular(L, C.T, upper=False)
    lam, Q = torch.linalg.eigh(0.5 * (C + C.T))
    return lam, torch.linalg.solve_triangular(L.T, Q, upper=True)


def _eigenvalue_sum(lams):
    out = torch.zeros(1, dtype=torch.float64, device="cuda")
    for v in lams[::-1]:
        out = (out[:, None] + v[None, :]).reshape(-1)
    return out


def _inside(n):
    """Flat mask of the nodes inside the box (no first or last node of any direction)."""
    keep = torch.ones(1, dtype=torch.bool, device="cuda")
    for v in n[::-1]:
        m = torch.ones(v, dtype=torch.bool, device="cuda")
        m[0] = m[-1] = False
        keep = (keep[:, None] & m[None, :]).reshape(-1)
    return keep


class _FD:
    """Fast diagonalisation in FP64: U (1 / Lambda) U^T on the inner nodes."""

    def __init__(self, p, elements):
        pairs = [_eigenpairs(p, ne) for ne in elements]
        self.U = [u for _, u in pairs]
        self.lam = _eigenvalue_sum([v for v, _ in pairs])
        self.keep = _inside([ne + p for ne in elements])

    def __call__(self, x):
        y = torch.zeros_like(x)
        t = _kron([u.T.contiguous() for u in self.U], x[self.keep]) / self.lam
        y[self.keep] = _kron(self.U, t)
        return y


def _solution(p, elements, coefs, b):
    """A x = b on the inner nodes by preconditioned GMRES with restarts, iterated to
    rounding."""
    rules = _rules(p, elements)
    B, W = _dense_rules(rules)
    P = _FD(p, elements)
    keep = P.keep.double()
    b = b * keep

    def A(v):
        return _product(B, W, coefs, "gradu_gradv", 3, False, v) * keep

    x = torch.zeros_like(b)
    for _ in range(3):
        r = b - A(x)
        beta = float(r.norm())
        V, Z, H = [r / beta], [], np.zeros((13, 12))
        for j in range(12):
            Z.append(P(V[j]))
            w = A(Z[j])
            for _ in range(2):
                for i, v in enumerate(V):
                    h = float(v @ w)
                    H[i, j] += h
                    w = w - h * v
            H[j + 1, j] = float(w.norm())
            V.append(w / H[j + 1, j])
        rhs = np.zeros(13)
        rhs[0] = beta
        y = np.linalg.lstsq(H, rhs, rcond=None)[0]
        for c, z in zip(y, Z):
            x = x + float(c) * z
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        parts = []
        for i, (p, ne) in enumerate(_batch_layout(case)):
            rules = _rules(p, [ne] * 3)
            coefs = _coefficients(rules, "gradu_gradv", 3, seed + i, torch.float64)
            b = _vector(_sizes(rules)[0], seed + i, torch.float64)
            parts.append(_solution(p, [ne] * 3, coefs, b))
        return torch.cat(parts)
    p, elements = case["p"], _elements(case)
    ndim = len(elements)
    dtype = DTYPES[case.get("dtype", "f64")]
    rules = _rules(p, elements, case.get("rule", "wq2"))
    n = _sizes(rules)[0]
    if kind == "geometry":
        B, _ = _dense_rules(rules)
        P = _ctrlpts(p, elements, seed)
        J = torch.stack([torch.stack([_kron([B[d][int(d == j)] for d in range(3)], c)
                                      for j in range(3)]) for c in P])
        cof = torch.stack([torch.linalg.cross(J[:, (j + 1) % 3], J[:, (j + 2) % 3], dim=0)
                           for j in range(3)])
        det = (J[:, 0] * cof[0]).sum(0)
        del J
        C = torch.stack([torch.stack([(cof[i] * cof[j]).sum(0) / det for j in range(3)])
                         for i in range(3)])
        return {"stiffness": C, "mass": det}
    if kind == "matvec":
        spd = ndim - 1 if case["st"] else ndim
        coefs = _coefficients(rules, case["op"], spd, seed, dtype)
        x = _vector(n, seed, dtype, case["cols"]).double()
        B, W = _dense_rules(rules)
        if case["cols"] == 1:
            return _product(B, W, coefs, case["op"], spd, case["st"], x)
        return torch.stack([_product(B, W, coefs, case["op"], spd, case["st"], x[:, k])
                            for k in range(case["cols"])], dim=1)
    if kind == "solve":
        coefs = _coefficients(rules, "gradu_gradv", 3, seed, torch.float64)
        return _solution(p, elements, coefs, _vector(n, seed, torch.float64))
    x = _vector(n, seed, dtype).double()
    if kind in ("fd", "fd_tc"):
        return _FD(p, elements)(x)
    # space-time: (advection in time) x (mass in space) + (mass in time) x (stiffness in
    # space), diagonal in space after the generalized eigenvectors
    space = _FD(p, elements[:-1])
    M, _, D = _pencil(p, elements[-1])
    M, D = M[1:, 1:], D[1:, 1:]
    nt = elements[-1] + p
    t = x.reshape(nt, -1)[1:, space.keep]
    t = torch.stack([_kron([u.T.contiguous() for u in space.U], r) for r in t])
    A = D[None, :, :] + space.lam[:, None, None] * M[None, :, :]
    z = torch.linalg.solve(A, t.T.unsqueeze(-1)).squeeze(-1).T
    y = torch.zeros((nt, space.keep.numel()), dtype=torch.float64, device="cuda")
    inner = torch.stack([_kron(space.U, r) for r in z.contiguous()])
    y[1:, space.keep] = inner
    return y.reshape(-1)
