"""Workloads of the Schwarz-smoother library, each one a call (or two) of its Python interface.

Families (`kind`):

  smoother    SchwarzPreconditioner.vmult on one Cartesian level: additive and multiplicative,
              vertex and cell patches, FP64 and FP32 arithmetic
  step        SchwarzSmoother.step, x += damping P (b - A x), on a Cartesian or distorted level
  operator    LaplaceOperator.vmult / vmult_fp32 on a Cartesian or distorted level
  transfer    prolongate_add and restrict_add between two levels
  vcycle      MultigridSolver.vmult, the preconditioner application of a CG solve
  solve       MultigridSolver.solve
  c0ip        C0IPBiharmonic.vmult and .smooth on the finest level
  mlp         MLP.forward and MLP.loss_grad of the learned local solver's network

Vectors are float64 device tensors in the library's DoF numbering: cells lexicographic (x
fastest), (k+1)^dim lexicographic DoFs per cell. `exact` evaluates the same linear maps in 64 bits
with torch and numpy from their definitions (1-D SIPG matrices, generalized eigenproblems,
quadrature on multilinear cells).
"""
import math

import numpy as np
import torch

import tpss_gb300 as tpss
from tpss_gb300.mesh import distorted_cube

DEV = "cuda"
F64 = torch.float64
DAMPING = {2: 0.25, 3: 0.15}  # the library's damping of additive vertex patches


# ---------------------------------------------------------------------------------------------
# the listed cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # a coarse multigrid level: the smallest smoother call, a few microseconds of work per color
        dict(name="smooth64_2d_k3_16", kind="smoother", dim=2, degree=3, nx=16, ny=16, nz=1, patch="vertex",
             variant="additive", precision="fp64"),
        # the 2D benchmark level (SIPG DGQ3, 64 x 64 cells) in single-precision smoother arithmetic
        dict(name="smooth32_2d_k3_64", kind="smoother", dim=2, degree=3, nx=64, ny=64, nz=1, patch="vertex",
             variant="additive", precision="fp32"),
        # the default (FP64) smoother on an ordinary 3D level
        dict(name="smooth64_3d_k4_40", kind="smoother", dim=3, degree=4, nx=40, ny=40, nz=40, patch="vertex",
             variant="additive", precision="fp64"),
        # the headline level (SIPG DGQ4, 64^3 cells, 32.8 M DoFs), FP32 smoother: the largest case
        dict(name="smooth32_3d_k4_64", kind="smoother", dim=3, degree=4, nx=64, ny=64, nz=64, patch="vertex",
             variant="additive", precision="fp32"),
        # one Richardson sweep on a level whose sizes divide nothing
        dict(name="step64_3d_k3_33x26x21", kind="step", dim=3, degree=3, nx=33, ny=26, nz=21, precision="fp64",
             distortion=0.0),
        # multiplicative vertex patches: a residual with the level operator between the colors
        dict(name="mult64_2d_k4_48", kind="smoother", dim=2, degree=4, nx=48, ny=48, nz=1, patch="vertex",
             variant="multiplicative", precision="fp64"),
        # the outer CG's operator product on the headline level
        dict(name="operator64_3d_k4_64", kind="operator", dim=3, degree=4, nx=64, ny=64, nz=64, precision="fp64",
             distortion=0.0),
        # one V-cycle in the recommended precision: FP32 smoothers, FP64 operators and transfers
        dict(name="vcycle32_3d_k4_32", kind="vcycle", dim=3, degree=4, cells=32, precision="fp32",
             vcycle_precision="fp64"),
        # a small 2D solve, every kernel a few microseconds; a loose tolerance, as for an inner solve
        dict(name="solve64_2d_k3_64", kind="solve", dim=2, degree=3, cells=64, precision="fp64"),
        # a Richardson sweep on distorted hexahedra (mapped operator, surrogate patches)
        dict(name="step64_3d_k3_20_distorted", kind="step", dim=3, degree=3, nx=20, ny=20, nz=20, precision="fp64",
             distortion=0.15),
        # the biharmonic benchmark level (C0IP Q3, 256 x 256 cells): operator and FP32 smoother
        dict(name="c0ip_2d_q3_256", kind="c0ip", degree=3, cells=256, precision="fp32", local="fd"),
        # gradients of the learned local solver's network on the patches of a 32^3 mesh
        dict(name="mlp_87x64x108_29791", kind="mlp", n_in=87, n_out=108, hidden=64, layers=3, rows=29791),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(rng, dim, degree, lo_dofs, hi_dofs, least=2):
    """Cells per direction (unequal, odd ones among them) for about a log-uniform number of DoFs."""
    dofs = math.exp(rng.uniform(math.log(lo_dofs), math.log(hi_dofs)))
    n = (dofs ** (1.0 / dim)) / (degree + 1)
    c = [max(least, int(round(n * rng.uniform(0.75, 1.33)))) for _ in range(dim)]
    return dict(nx=c[0], ny=c[1], nz=c[2] if dim == 3 else 1)


def draw(rng):
    kind = rng.choice(["smoother"] * 4 + ["step"] * 2 + ["operator"] * 2 + ["transfer", "vcycle", "vcycle", "solve",
                                                                           "c0ip", "mlp"])
    dim = rng.choice([2, 3])
    # degrees 1..7; in 3D mostly the low ones, as the configurations use
    degree = rng.choice([1, 2, 3, 4, 5, 6, 7] if dim == 2 else [1, 2, 2, 3, 3, 4, 4, 5, 6, 7])
    precision = rng.choice(["fp64", "fp64", "fp32"])
    if kind == "smoother":
        patch = rng.choice(["vertex", "vertex", "vertex", "cell"])
        variant = rng.choice(["additive", "additive", "additive", "multiplicative"])
        hi = 4e6 if variant == "additive" else 5e5
        return dict(kind=kind, dim=dim, degree=degree, patch=patch, variant=variant, precision=precision,
                    **_cells(rng, dim, degree, 2e3, hi))
    if kind in ("step", "operator"):
        distortion = rng.choice([0.0, 0.0, 0.15])
        if distortion:
            degree = min(degree, 3 if dim == 3 else 5)
        hi = 4e6 if not distortion else 3e5
        return dict(kind=kind, dim=dim, degree=degree, precision=precision, distortion=distortion,
                    **_cells(rng, dim, degree, 2e3, hi))
    if kind == "transfer":
        return dict(kind=kind, dim=dim, degree=degree, precision="fp64", **_cells(rng, dim, degree, 1e3, 5e5, 1))
    if kind in ("vcycle", "solve"):
        most = {2: 128, 3: 32 if degree <= 3 else 16}[dim] // (1 if kind == "vcycle" else 2)
        cells = 2 ** rng.randint(2, int(math.log2(most))) * rng.choice([1, 1, 3])
        cells = cells if cells <= most else cells // 3
        c = dict(kind=kind, dim=dim, degree=degree, cells=cells, precision=precision if kind == "vcycle" else "fp64")
        if kind == "vcycle":
            c["vcycle_precision"] = "fp64" if precision == "fp64" else rng.choice(["fp64", "fp32"])
        return c
    if kind == "c0ip":
        degree = rng.randint(2, 5)
        return dict(kind=kind, degree=degree, cells=2 ** rng.randint(3, 8 if degree < 4 else 7),
                    precision=rng.choice(["fp64", "fp32"]), local=rng.choice(["fd", "exact"]))
    n = 2 * (rng.randint(1, 3) + 1)  # patch size per direction: degrees 1..3
    return dict(kind="mlp", n_in=3 ** dim * dim + 2 * dim, n_out=dim * n * (n + 1) // 2, hidden=rng.choice([32, 64, 96]),
                layers=rng.randint(1, 3), rows=_log_int(rng, 200, 30000))


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _nc(c):
    return [c["nx"], c["ny"], c["nz"]][: c["dim"]]


def _n_dofs(c):
    return math.prod(_nc(c)) * (c["degree"] + 1) ** c["dim"]


def _uniform(n, seed, k=0):
    """A load or residual: f ~ U[-1, 1] per DoF."""
    g = torch.Generator(device=DEV)
    g.manual_seed(1000003 * seed + 17 * k + 1)
    return torch.rand(n, generator=g, device=DEV, dtype=F64) * 2.0 - 1.0


def _smooth(n, seed, k=0):
    """An iterate: a slowly varying part and a rough one a hundred times smaller."""
    t = torch.arange(n, device=DEV, dtype=F64) / n
    r = _uniform(8, seed, 100 + k)
    s = sum(r[i] * torch.sin((3.0 * i + 2.0) * t + r[i + 4]) for i in range(4))
    return s + 0.01 * _uniform(n, seed, k)


def _prec(name):
    return tpss.Precision.fp64 if name == "fp64" else tpss.Precision.fp32


def _coords(c, seed):
    return distorted_cube(c["dim"], _nc(c), seed, c["distortion"])


def _layout(c, seed, patch="vertex", variant="additive"):
    AD = tpss.SubdomainHandler.AdditionalData
    ad = AD(dim=c["dim"], degree=c["degree"], n_cells=_nc(c), patch_variant=getattr(tpss.PatchVariant, patch),
            smoother_variant=getattr(tpss.SmootherVariant, variant))
    if c.get("distortion"):
        ad.vertex_coords = _coords(c, seed)
    return tpss.SubdomainHandler(ad)


def _relaxation(c):
    return tpss.lookup_damping_factor(getattr(tpss.PatchVariant, c.get("patch", "vertex")),
                                      getattr(tpss.SmootherVariant, c.get("variant", "additive")), c["dim"])


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state["kind"]](state)


def _prepare_smoother(c, seed):
    sh = _layout(c, seed, c["patch"], c["variant"])
    op = tpss.LaplaceOperator(sh) if c["variant"] == "multiplicative" else None
    p = tpss.SchwarzPreconditioner()
    p.initialize(sh, op, tpss.SchwarzPreconditioner.AdditionalData(relaxation=_relaxation(c),
                                                                   precision=_prec(c["precision"])))
    src = _uniform(sh.n_dofs(), seed)
    return dict(kind="smoother", layout=sh, op=op, p=p, src=src, dst=torch.empty_like(src))


def _run_smoother(s):
    s["p"].vmult(s["dst"], s["src"])
    return s["dst"]


def _prepare_step(c, seed):
    sh = _layout(c, seed)
    op = tpss.LaplaceOperator(sh)
    p = tpss.SchwarzPreconditioner()
    p.initialize(sh, op, tpss.SchwarzPreconditioner.AdditionalData(relaxation=_relaxation(c) * (0.5 if c["distortion"] else 1.0),
                                                                   precision=_prec(c["precision"])))
    sm = tpss.SchwarzSmoother()
    sm.initialize(op, p)
    n = sh.n_dofs()
    return dict(kind="step", layout=sh, op=op, p=p, smoother=sm, x=_smooth(n, seed), b=_uniform(n, seed, 1))


def _run_step(s):
    s["smoother"].step(s["x"], s["b"])
    return s["x"]


def _prepare_operator(c, seed):
    sh = _layout(c, seed)
    op = tpss.LaplaceOperator(sh)
    src = _smooth(sh.n_dofs(), seed)
    return dict(kind="operator", layout=sh, op=op, src=src, dst=torch.empty_like(src), precision=c["precision"])


def _run_operator(s):
    if s["precision"] == "fp64":
        s["op"].vmult(s["dst"], s["src"])
    else:
        s["op"].vmult_fp32(s["dst"], s["src"])
    return s["dst"]


def _prepare_transfer(c, seed):
    n = _n_dofs(c)
    nf = n * 2 ** c["dim"]
    return dict(kind="transfer", dim=c["dim"], degree=c["degree"], nc=_nc(c), coarse=_smooth(n, seed),
                fine=_smooth(nf, seed, 1), coarse_r=_uniform(n, seed, 2), fine_r=_uniform(nf, seed, 3))


def _run_transfer(s):
    tpss.prolongate_add(s["dim"], s["degree"], s["nc"], s["fine"], s["coarse"])
    tpss.restrict_add(s["dim"], s["degree"], s["nc"], s["coarse_r"], s["fine_r"])
    return s["fine"], s["coarse_r"]


def _roots(cells):
    """Root cells per direction of a mesh with `cells` = roots * 2^L cells (one or three roots)."""
    return 3 if cells % 3 == 0 else 1


def _multigrid(c):
    return tpss.MultigridSolver(c["dim"], c["degree"], _roots(c["cells"]), c["cells"], precision=_prec(c["precision"]),
                                vcycle_precision=_prec(c.get("vcycle_precision", "fp64")), coarse_solver=1)


def _prepare_vcycle(c, seed):
    mg = _multigrid(c)
    src = _uniform(mg.n_dofs(), seed)
    return dict(kind="vcycle", mg=mg, src=src, dst=torch.empty_like(src))


def _run_vcycle(s):
    s["mg"].vmult(s["dst"], s["src"])
    return s["dst"]


SOLVE_TOL = 1e-4


def _prepare_solve(c, seed):
    mg = _multigrid(c)
    f = _uniform(mg.n_dofs(), seed)
    return dict(kind="solve", mg=mg, f=f, u=torch.empty_like(f))


def _run_solve(s):
    its, history = s["mg"].solve(s["u"], s["f"], rel_tol=SOLVE_TOL)
    return its, history, s["u"]


def _prepare_c0ip(c, seed):
    p = tpss.C0IPBiharmonic(c["degree"], 2, c["cells"], local_solver=0 if c["local"] == "fd" else 1,
                            precision=_prec(c["precision"]), relaxation=DAMPING[2])
    n = p.n_dofs()
    u, f = _smooth(n, seed), _uniform(n, seed, 1)
    return dict(kind="c0ip", p=p, u=u, f=f, Au=torch.empty_like(u), Pf=torch.empty_like(u))


def _run_c0ip(s):
    s["p"].vmult(s["Au"], s["u"])
    s["p"].smooth(s["Pf"], s["f"])
    return s["Au"], s["Pf"]


def _widths(c):
    return [c["n_in"]] + [c["hidden"]] * c["layers"] + [c["n_out"]]


def _mlp_data(c, seed):
    rng = np.random.Generator(np.random.Philox(seed))
    w = _widths(c)
    params = []
    for a, b in zip(w[:-1], w[1:]):  # Glorot-uniform weights, small biases
        params += [rng.uniform(-1, 1, b * a) * math.sqrt(6.0 / (a + b)), 0.05 * rng.uniform(-1, 1, b)]
    params = np.concatenate(params).astype(np.float32)
    x = (0.2 * _uniform(c["rows"] * c["n_in"], seed)).float().reshape(c["rows"], c["n_in"])
    t = (0.1 * _uniform(c["rows"] * c["n_out"], seed, 1)).float().reshape(c["rows"], c["n_out"])
    return params, x, t


def _prepare_mlp(c, seed):
    params, x, t = _mlp_data(c, seed)
    m = tpss.MLP(c["n_in"], c["n_out"], c["hidden"], c["layers"])
    m.set_params(params)
    return dict(kind="mlp", m=m, x=x, t=t)


def _run_mlp(s):
    y = s["m"].forward(s["x"])
    loss, grad = s["m"].loss_grad(s["x"], s["t"])
    return y, loss, grad


_PREPARE = dict(smoother=_prepare_smoother, step=_prepare_step, operator=_prepare_operator, transfer=_prepare_transfer,
                vcycle=_prepare_vcycle, solve=_prepare_solve, c0ip=_prepare_c0ip, mlp=_prepare_mlp)
_RUN = dict(smoother=_run_smoother, step=_run_step, operator=_run_operator, transfer=_run_transfer, vcycle=_run_vcycle,
            solve=_run_solve, c0ip=_run_c0ip, mlp=_run_mlp)


# ---------------------------------------------------------------------------------------------
# bytes and operations of one pass
# ---------------------------------------------------------------------------------------------
def _smoother_flops(dim, degree, nc, ncp):
    """2 d passes of an n x n contraction per patch, halved by the mirror symmetry, and the division."""
    n = ncp * (degree + 1)
    patches = math.prod(max(0, m - ncp + 1) for m in nc)
    return patches * (2 * dim * n ** (dim + 1) + 2 * n ** dim)


def _operator_flops(dim, degree, nc):
    """Per direction the cell's 1-D block and two rank-2 couplings, then the shared mass passes."""
    n = degree + 1
    passes = {2: 4, 3: 8}[dim]
    return math.prod(nc) * n ** dim * (2 * n * passes + 8 * dim)


def _mapped_flops(dim, degree, nc):
    n = degree + 1
    return math.prod(nc) * n ** dim * (4 * dim * n + 2 * 2 * dim * 12)


def _vcycle_work(c):
    dim, k = c["dim"], c["degree"]
    n, byts, flops = c["cells"], 0, 0
    while n > _roots(c["cells"]):
        N = n ** dim * (k + 1) ** dim
        # two smoothings, two residuals (level vectors in and out) and the transfers
        byts += N * 8 * (2 * 2 + 2 * 3 + 2)
        flops += 2 * _smoother_flops(dim, k, [n] * dim, 2) + 2 * _operator_flops(dim, k, [n] * dim) + 8 * dim * (k + 1) * N
        n //= 2
    return byts, flops


def work(case):
    c, kind = case, case["kind"]
    if kind in ("smoother", "step", "operator"):
        N, nc = _n_dofs(c), _nc(c)
        fs = _smoother_flops(c["dim"], c["degree"], nc, 1 if c.get("patch") == "cell" else 2)
        fo = (_mapped_flops if c.get("distortion") else _operator_flops)(c["dim"], c["degree"], nc)
        if kind == "operator":
            return dict(bytes=16 * N, flops=fo)
        if kind == "step":
            return dict(bytes=24 * N, flops=fs + fo)
        if c["variant"] == "additive":
            return dict(bytes=16 * N, flops=fs)
        colors = 2 ** c["dim"] if c["patch"] == "vertex" else 2
        return dict(bytes=16 * N, flops=fs + (colors - 1) * fo)
    if kind == "transfer":
        N = _n_dofs(c)
        return dict(bytes=8 * N * 3 + 8 * N * 2 ** c["dim"] * 3, flops=4 * c["dim"] * (c["degree"] + 1) * N * 2 ** c["dim"])
    if kind == "vcycle":
        b, f = _vcycle_work(c)
        return dict(bytes=b, flops=f)
    if kind == "solve":
        b, f = _vcycle_work(c)
        N = c["cells"] ** c["dim"] * (c["degree"] + 1) ** c["dim"]
        its = 8
        return dict(bytes=its * (b + 8 * 8 * N), flops=its * (f + _operator_flops(c["dim"], c["degree"], [c["cells"]] * c["dim"])))
    if kind == "c0ip":
        N, m = (c["cells"] * c["degree"] - 1) ** 2, 2 * c["degree"] - 1
        patches = (c["cells"] - 1) ** 2
        fs = patches * (8 * m ** 3 if c["local"] == "fd" else 2 * m ** 4)
        return dict(bytes=32 * N, flops=fs + N * 2 * 2 * (8 * c["degree"] + 3))
    w = _widths(c)
    macs = sum(a * b for a, b in zip(w[:-1], w[1:]))
    return dict(bytes=4 * c["rows"] * (c["n_in"] + 2 * c["n_out"]) + 8 * macs, flops=2 * c["rows"] * macs * 4)


# ---------------------------------------------------------------------------------------------
# the same maps in 64 bits, from their definitions
# ---------------------------------------------------------------------------------------------
def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return 0.5 * (x + 1.0), 0.5 * w


def _lobatto(n):
    """Gauss-Lobatto points on [0, 1]: the end points and the roots of P'_(n-1)."""
    c = np.zeros(n)
    c[n - 1] = 1.0
    d = np.polynomial.legendre.legder(c)
    x = np.sort(np.real(np.polynomial.legendre.legroots(d)))
    dd = np.polynomial.legendre.legder(d)
    x = x - np.polynomial.legendre.legval(x, d) / np.polynomial.legendre.legval(x, dd) if x.size else x
    return np.concatenate([[0.0], 0.5 * (x + 1.0), [1.0]])


def _lagrange(z, x):
    """Values, first and second derivatives [basis, point] of the Lagrange basis on z."""
    n = len(z)
    V, D, E = np.zeros((n, len(x))), np.zeros((n, len(x))), np.zeros((n, len(x)))
    for i in range(n):
        f, f1, f2 = np.ones(len(x)), np.zeros(len(x)), np.zeros(len(x))
        for j in range(n):
            if j != i:
                t = 1.0 / (z[i] - z[j])
                f2 = f2 * (x - z[j]) * t + 2 * f1 * t
                f1 = f1 * (x - z[j]) * t + f * t
                f = f * (x - z[j]) * t
        V[i], D[i], E[i] = f, f1, f2
    return V, D, E


def _dg_1d(k, h):
    """Global 1-D DG mass and SIPG matrices on cells of widths h."""
    np_, nc = k + 1, len(h)
    z = _lobatto(np_)
    qx, qw = _gauss(np_)
    V, D, _ = _lagrange(z, qx)
    F, G, _ = _lagrange(z, np.array([0.0, 1.0]))
    M, A = np.zeros((nc * np_, nc * np_)), np.zeros((nc * np_, nc * np_))
    gamma = k * (k + 1.0)
    for c in range(nc):
        s = slice(c * np_, (c + 1) * np_)
        M[s, s] += (V * qw) @ V.T * h[c]
        A[s, s] += (D * qw) @ D.T / h[c]
    for f in range(nc + 1):
        # jump and mean normal derivative of every basis function at face f
        jump, mean, idx = [], [], []
        inner = 0 < f < nc
        if f > 0:
            idx += range((f - 1) * np_, f * np_)
            jump += list(F[:, 1])
            mean += list(G[:, 1] / h[f - 1] * (0.5 if inner else 1.0))
        if f < nc:
            idx += range(f * np_, (f + 1) * np_)
            jump += list(-F[:, 0])
            mean += list(G[:, 0] / h[f] * (0.5 if inner else 1.0))
        j, m = np.array(jump), np.array(mean)
        sigma = gamma * 0.5 * (1 / h[f - 1] + 1 / h[f]) if inner else 2 * gamma / (h[0] if f == 0 else h[-1])
        A[np.ix_(idx, idx)] += sigma * np.outer(j, j) - np.outer(m, j) - np.outer(j, m)
    return M, A


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device=DEV)


def _grid(u, nc, np_):
    """Library numbering -> tensor over the global 1-D indices (z, y, x)."""
    dim = len(nc)
    r = list(reversed(nc))
    u = u.reshape(r + [np_] * dim)
    perm = [i for d in range(dim) for i in (d, dim + d)]
    return u.permute(perm).reshape([n * np_ for n in r]).contiguous()


def _ungrid(g, nc, np_):
    dim = len(nc)
    r = list(reversed(nc))
    g = g.reshape([m for n in r for m in (n, np_)])
    perm = [2 * d for d in range(dim)] + [2 * d + 1 for d in range(dim)]
    return g.permute(perm).reshape(-1).contiguous()


def _along(B, g, axis):
    """(I x .. x B x .. x I) g along an axis of the tensor."""
    return torch.movedim(torch.matmul(B, torch.movedim(g, axis, -2)), -2, axis) if g.dim() > 1 else B @ g


class _Level:
    """The SIPG operator, patch solver and mesh data of one Cartesian level (unit cube)."""

    def __init__(self, dim, k, nc):
        self.dim, self.k, self.nc, self.np = dim, k, list(nc), k + 1
        pairs = [_dg_1d(k, [1.0 / n] * n) for n in nc]
        self.M = [p[0] for p in pairs]
        self.A = [p[1] for p in pairs]
        self.Mt, self.At = [_dev(m) for m in self.M], [_dev(a) for a in self.A]

    def axis(self, d):
        return self.dim - 1 - d

    def apply(self, g):
        out = torch.zeros_like(g)
        for d in range(self.dim):
            t = _along(self.At[d], g, self.axis(d))
            for e in range(self.dim):
                if e != d:
                    t = _along(self.Mt[e], t, self.axis(e))
            out += t
        return out

    def eigen(self, d, ncp):
        """Generalized eigenvectors and eigenvalues of the 1-D patch problems of direction d."""
        n, S, lam = ncp * self.np, [], []
        for c in range(self.nc[d] - ncp + 1):
            if 2 <= c < self.nc[d] - ncp - 1:
                S.append(S[-1])
                lam.append(lam[-1])
                continue
            s = slice(c * self.np, c * self.np + n)
            s_, l_ = _gen_eig(self.M[d][s, s], self.A[d][s, s])
            S.append(s_)
            lam.append(l_)
        return _dev(np.array(S)).reshape(-1, n, n), _dev(np.array(lam)).reshape(-1, n)

    def smooth(self, g, omega, ncp=2, color=None):
        """omega sum_j R_j^T A_j^-1 R_j g, over all patches or over those of one color."""
        dim, np_, out = self.dim, self.np, torch.zeros_like(g)
        n = ncp * np_
        if min(self.nc) < ncp:
            return out
        eig = [self.eigen(d, ncp) for d in range(dim)]
        starts = []
        for d in range(dim):
            a = torch.arange(self.nc[d] - ncp + 1)
            if color is not None and ncp == 2:
                a = a[a % 2 == (color >> d) & 1]
            starts.append(a)
        if any(len(a) == 0 for a in starts):
            return out
        top = starts[dim - 1]
        per = max(1, int(3e7 / (math.prod(len(a) for a in starts[: dim - 1]) * n ** dim)))
        for part in torch.split(top, per):
            use = starts[: dim - 1] + [part]
            w = g
            for d in reversed(range(dim)):  # windows [P_z, P_y, P_x, n_z, n_y, n_x]
                w = w.unfold(self.axis(d), n, np_)
                w = w.index_select(self.axis(d), use[d].to(DEV))
            w = w.contiguous()
            S = [eig[d][0][use[d].to(DEV)] for d in range(dim)]
            lam = [eig[d][1][use[d].to(DEV)] for d in range(dim)]
            w = _kron_windows([s.transpose(1, 2) for s in S], w)
            if dim == 3:
                den = lam[2][:, None, None, :, None, None] + lam[1][None, :, None, None, :, None] + lam[0][None, None, :, None, None, :]
            else:
                den = lam[1][:, None, :, None] + lam[0][None, :, None, :]
            if color is not None and ncp == 1:
                odd = [(use[d].to(DEV) % 2) for d in range(dim)]
                par = (odd[1][:, None] + odd[0][None, :]) if dim == 2 else (odd[2][:, None, None] + odd[1][None, :, None] + odd[0][None, None, :])
                w = w * (par % 2 == color).to(F64)[(...,) + (None,) * dim]
            w = omega * _kron_windows(S, w / den)
            _scatter_windows(out, w, use, ncp, np_, self)
        return out


def _gen_eig(M, A):
    L = np.linalg.cholesky(M)
    Li = np.linalg.inv(L)
    lam, Q = np.linalg.eigh(Li @ A @ Li.T)
    return Li.T @ Q, lam


def _kron_windows(S, w):
    """Apply S[d][patch position] along direction d of every window."""
    if w.dim() == 6:
        w = torch.einsum("xij,zyxabj->zyxabi", S[0], w)
        w = torch.einsum("yij,zyxajc->zyxaic", S[1], w)
        return torch.einsum("zij,zyxjbc->zyxibc", S[2], w)
    w = torch.einsum("xij,yxaj->yxai", S[0], w)
    return torch.einsum("yij,yxja->yxia", S[1], w)


def _along_batch(B, w, axis):
    """B[p] along an axis of w[p]."""
    t = torch.movedim(w, axis, -1)
    r = torch.matmul(t.reshape(t.shape[0], -1, t.shape[-1]), B.transpose(1, 2)).reshape(t.shape)
    return torch.movedim(r, -1, axis)


def _scatter_windows(out, w, use, ncp, np_, level):
    dim = level.dim
    cells = out.reshape([m for d in reversed(range(dim)) for m in (level.nc[d], np_)])
    use = [u.to(DEV) for u in use]
    for b in range(ncp ** dim):
        off = [(b // ncp ** d) % ncp for d in range(dim)]
        part = w
        for d in range(dim):
            ax = dim + level.axis(d)
            part = part.narrow(ax, off[d] * np_, np_)
        idx = [use[d] + off[d] for d in range(dim)]
        if dim == 3:
            p = part.permute(0, 3, 1, 4, 2, 5)
            cells[idx[2][:, None, None], :, idx[1][None, :, None], :, idx[0][None, None, :], :] += p.permute(0, 2, 4, 1, 3, 5)
        else:
            cells[idx[1][:, None], :, idx[0][None, :], :] += part


def _embed(k, n):
    """1-D embedding of the DG space on n cells into the one on 2 n cells."""
    z = _lobatto(k + 1)
    E = np.zeros((2 * n * (k + 1), n * (k + 1)))
    for s in range(2):
        V, _, _ = _lagrange(z, 0.5 * (z + s))
        for c in range(n):
            E[(2 * c + s) * (k + 1): (2 * c + s + 1) * (k + 1), c * (k + 1): (c + 1) * (k + 1)] = V.T
    return _dev(E)


def _all_axes(mats, g):
    for d, B in enumerate(mats):
        g = _along(B, g, len(mats) - 1 - d)
    return g


def _exact_vcycle(c, g):
    dim, k, omega = c["dim"], c["degree"], DAMPING[c["dim"]]

    def cycle(n, b):
        lv = _Level(dim, k, [n] * dim)
        if n == _roots(c["cells"]):
            N = b.numel()
            A = torch.stack([lv.apply(e.reshape(b.shape)).reshape(-1) for e in torch.eye(N, dtype=F64, device=DEV)], 1)
            return torch.linalg.solve(A, b.reshape(-1)).reshape(b.shape)
        E = _embed(k, n // 2)
        x = lv.smooth(b, omega)
        x = x + _all_axes([E] * dim, cycle(n // 2, _all_axes([E.T] * dim, b - lv.apply(x))))
        return x + lv.smooth(b - lv.apply(x), omega)

    return cycle(c["cells"], g)


class _Mapped:
    """SIPG operator and surrogate patches of a level with multilinear cells, by quadrature."""

    def __init__(self, dim, k, nc, X):
        self.dim, self.k, self.nc, self.np = dim, k, list(nc), k + 1
        nv = [n + 1 for n in nc]
        V = torch.as_tensor(X, dtype=F64, device=DEV).reshape(list(reversed(nv)) + [dim])
        corners = []
        for b in range(2 ** dim):
            sl = tuple(slice((b >> d) & 1, ((b >> d) & 1) + nc[d]) for d in reversed(range(dim)))
            corners.append(V[sl])
        self.X = torch.stack(corners, dim=dim)  # [nz, ny, nx, corner, dim]
        z = _lobatto(k + 1)
        self.qx, self.qw = _gauss(k + 1)
        self.q = _lagrange(z, self.qx)[:2]
        self.f = _lagrange(z, np.array([0.0, 1.0]))[:2]

    def jac_inv(self, X, xi):
        """J^-1 and det J [cells.., points, dim, dim] at the points xi [points, dim]."""
        dim, xi = self.dim, _dev(xi)
        W = []
        for b in range(2 ** dim):
            row = []
            for j in range(dim):
                t = torch.ones(xi.shape[0], dtype=F64, device=DEV)
                for e in range(dim):
                    up = (b >> e) & 1
                    t = t * ((1.0 if up else -1.0) if e == j else (xi[:, e] if up else 1.0 - xi[:, e]))
                row.append(t)
            W.append(torch.stack(row, -1))
        W = torch.stack(W, 1)  # [points, corner, dim]
        J = torch.einsum("...ca,pcj->...paj", X, W)
        return torch.linalg.inv(J), torch.linalg.det(J)

    def basis(self, sides):
        """Basis values [points, dofs] and reference gradients [points, dofs, dim], points in the
        Gauss grid of the free directions; sides: {direction: face side}."""
        dim = self.dim
        v1 = [_dev(self.f[0][:, [sides[d]]] if d in sides else self.q[0]) for d in range(dim)]
        d1 = [_dev(self.f[1][:, [sides[d]]] if d in sides else self.q[1]) for d in range(dim)]

        def kron(m):
            out = m[0]
            for d in range(1, dim):
                out = torch.einsum("ap,bq->abpq", m[d], out).reshape(m[d].shape[0] * out.shape[0], -1)
            return out.T.contiguous()

        val = kron(v1)
        grad = torch.stack([kron([d1[d] if d == g else v1[d] for d in range(dim)]) for g in range(dim)], -1)
        return val, grad

    def points(self, sides):
        dim = self.dim
        ax = [np.array([float(sides[d])]) if d in sides else self.qx for d in range(dim)]
        wt = [np.array([1.0]) if d in sides else self.qw for d in range(dim)]
        g = np.meshgrid(*reversed(ax), indexing="ij")
        w = np.ones(g[0].shape)
        for d, m in enumerate(reversed(np.meshgrid(*reversed(wt), indexing="ij"))):
            w = w * m
        return np.stack([g[dim - 1 - d].reshape(-1) for d in range(dim)], -1), _dev(w.reshape(-1))

    def apply(self, u):
        dim, nd, gamma = self.dim, self.np ** self.dim, self.k * (self.k + 1.0)
        shape = list(reversed(self.nc))
        u = u.reshape(shape + [nd])
        y = torch.zeros_like(u)
        xi, w = self.points({})
        val, grad = self.basis({})
        Ji, det = self.jac_inv(self.X, xi)
        gu = torch.einsum("...i,qij->...qj", u, grad)
        gx = torch.einsum("...qj,...qja->...qa", gu, Ji)
        y += torch.einsum("...qj,qij->...i", torch.einsum("...qja,...qa->...qj", Ji, gx) * (w * det.abs())[..., None], grad)
        for d in range(dim):
            ax, n = dim - 1 - d, self.nc[d]
            side = {}
            for s in (0, 1):
                xi, w = self.points({d: s})
                val, grad = self.basis({d: s})
                Ji, det = self.jac_inv(self.X, xi)
                ng = Ji[..., d, :].norm(dim=-1)
                nrm = (1.0 if s else -1.0) * Ji[..., d, :] / ng[..., None]
                cn = torch.einsum("...ea,...a->...e", Ji, nrm)  # J^-1 n, outward
                side[s] = dict(val=val, grad=grad, w=w * det.abs() * ng, cn=cn, h=1.0 / ng[..., 0],
                               u=torch.einsum("...i,qi->...q", u, val),
                               du=torch.einsum("...qe,...qe->...q", torch.einsum("...i,qie->...qe", u, grad), cn))

            def test(s, sl, a, b):
                """y += a phi_i + b d_n phi_i at the faces of side s of the cells sl."""
                t = side[s]
                y[sl] += torch.einsum("...q,qi->...i", a, t["val"]) + torch.einsum("...qe,qie->...i", b[..., None] * t["cn"][sl], t["grad"])

            def cells(lo, hi):
                return tuple(slice(lo, hi) if i == ax else slice(None) for i in range(dim))

            lo, hi = cells(0, n - 1), cells(1, n)
            L, R = side[1], side[0]
            sig = (gamma * 0.5 * (1 / L["h"][lo] + 1 / R["h"][hi]))[..., None]
            jump, mean, w = L["u"][lo] - R["u"][hi], 0.5 * (L["du"][lo] - R["du"][hi]), L["w"][lo]
            test(1, lo, w * (sig * jump - mean), -0.5 * w * jump)
            test(0, hi, w * (mean - sig * jump), 0.5 * w * jump)
            for s, sl in ((0, cells(0, 1)), (1, cells(n - 1, n))):
                t = side[s]
                sig = (2.0 * gamma / t["h"][sl])[..., None]
                test(s, sl, t["w"][sl] * (sig * t["u"][sl] - t["du"][sl]), -t["w"][sl] * t["u"][sl])
        return y.reshape(-1)

    def smooth(self, r, omega):
        """Additive vertex patches on surrogate Cartesian patches: the widths are the average arc
        lengths between opposite cell faces (straight lines on a multilinear cell)."""
        dim, np_ = self.dim, self.np
        z = _lobatto(5)
        wl = 2.0 / (5 * 4 * np.polynomial.legendre.legval(2 * z - 1, [0, 0, 0, 0, 1]) ** 2) * 0.5
        n = 2 * np_
        h = []
        for d in range(dim):
            others = [e for e in range(dim) if e != d]
            acc = 0.0
            for i in range(5 ** (dim - 1)):
                t, wt = {}, 1.0
                for j, e in enumerate(others):
                    t[e] = z[(i // 5 ** j) % 5]
                    wt *= wl[(i // 5 ** j) % 5]
                diff = 0.0
                for b in range(2 ** dim):
                    cw = 1.0 if (b >> d) & 1 else -1.0
                    for e in others:
                        cw *= t[e] if (b >> e) & 1 else 1.0 - t[e]
                    diff = diff + cw * self.X[..., b, :]
                acc = acc + wt * diff.norm(dim=-1)
            h.append(acc)  # [nz, ny, nx]
        P = [m - 1 for m in self.nc]
        out = torch.zeros_like(r).reshape(list(reversed(self.nc)) + [np_] * dim)
        u = r.reshape(out.shape)
        corner = []
        for b in range(2 ** dim):
            corner.append(tuple(slice((b >> d) & 1, ((b >> d) & 1) + P[d]) for d in reversed(range(dim))))
        S, lam = [], []
        for d in range(dim):
            w = []
            for s in (0, 1):
                w.append(sum(h[d][corner[b]] for b in range(2 ** dim) if (b >> d) & 1 == s) / 2 ** (dim - 1))
            pos = torch.arange(P[d], device=DEV).reshape([-1 if i == dim - 1 - d else 1 for i in range(dim)]).expand(w[0].shape)
            M, A = self.patch_1d(w[0].reshape(-1), w[1].reshape(-1), (pos == 0).reshape(-1), (pos == P[d] - 1).reshape(-1))
            Lc = torch.linalg.cholesky(M)
            B = torch.linalg.solve_triangular(Lc, A, upper=False)
            B = torch.linalg.solve_triangular(Lc, B.transpose(1, 2), upper=False)
            l_, Q = torch.linalg.eigh(0.5 * (B + B.transpose(1, 2)))
            S.append(torch.linalg.solve_triangular(Lc.transpose(1, 2), Q, upper=True))
            lam.append(l_)
        np1 = math.prod(P)
        w = torch.zeros([np1] + [n] * dim, dtype=F64, device=DEV)
        for b in range(2 ** dim):
            sl = tuple(slice(((b >> d) & 1) * np_, (((b >> d) & 1) + 1) * np_) for d in reversed(range(dim)))
            w[(slice(None),) + sl] = u[corner[b]].reshape([np1] + [np_] * dim)
        for d in range(dim):
            w = _along_batch(S[d].transpose(1, 2), w, dim - d)
        den = 0.0
        for d in range(dim):
            den = den + lam[d].reshape([np1] + [n if i == dim - 1 - d else 1 for i in range(dim)])
        w = w / den
        for d in range(dim):
            w = _along_batch(S[d], w, dim - d)
        for b in range(2 ** dim):
            sl = tuple(slice(((b >> d) & 1) * np_, (((b >> d) & 1) + 1) * np_) for d in reversed(range(dim)))
            out[corner[b]] += omega * w[(slice(None),) + sl].reshape(list(reversed(P)) + [np_] * dim)
        return out.reshape(-1)

    def patch_1d(self, h0, h1, lo, hi):
        """1-D two-cell patch matrices (mass, SIPG) with widths h0, h1 and boundary flags, batched."""
        np_, gamma = self.np, self.k * (self.k + 1.0)
        V, D = self.q
        F, G = _dev(self.f[0]), _dev(self.f[1])
        Mr, Kr = _dev((V * self.qw) @ V.T), _dev((D * self.qw) @ D.T)
        B = h0.shape[0]
        M = torch.zeros((B, 2 * np_, 2 * np_), dtype=F64, device=DEV)
        A = torch.zeros_like(M)
        hs = (h0, h1)
        for c in (0, 1):
            s = slice(c * np_, (c + 1) * np_)
            M[:, s, s] += Mr * hs[c][:, None, None]
            A[:, s, s] += Kr / hs[c][:, None, None]
        for c, f, flag in ((0, 0, lo), (1, 1, hi)):  # outer faces: physical, or half of an interior face
            s, h = slice(c * np_, (c + 1) * np_), hs[c]
            avg = torch.where(flag, 1.0, 0.5).to(F64)
            nu = 1.0 if f else -1.0
            v, g = F[:, f], nu * G[:, f]
            A[:, s, s] += (2 * gamma * avg / h)[:, None, None] * torch.outer(v, v) - (avg / h)[:, None, None] * (torch.outer(v, g) + torch.outer(g, v))
        j = torch.cat([F[:, 1], -F[:, 0]]).expand(B, -1)
        m = torch.cat([0.5 * G[:, 1][None] / h0[:, None], 0.5 * G[:, 0][None] / h1[:, None]], 1)
        # penalty of the patch interface: gamma / h of the own cell on the diagonal blocks, the mean
        # of both on the coupling blocks (FDEvaluation::patch_action)
        own = torch.cat([(gamma / h0)[:, None].expand(B, np_), (gamma / h1)[:, None].expand(B, np_)], 1)
        first = torch.arange(2 * np_, device=DEV) < np_
        sig = torch.where(first[:, None] == first[None, :], own[:, :, None], (gamma * 0.5 * (1 / h0 + 1 / h1))[:, None, None])
        A += sig * j[:, :, None] * j[:, None, :] - m[:, :, None] * j[:, None, :] - j[:, :, None] * m[:, None, :]
        return M, A


def _exact_smoother(c, seed):
    lv = _Level(c["dim"], c["degree"], _nc(c))
    ncp = 1 if c["patch"] == "cell" else 2
    omega = _relaxation_value(c)
    g = _grid(_uniform(_n_dofs(c), seed), _nc(c), lv.np)
    if c["variant"] == "additive":
        return _ungrid(lv.smooth(g, omega, ncp), _nc(c), lv.np)
    x = torch.zeros_like(g)
    for color in range(2 ** c["dim"] if ncp == 2 else 2):
        x = x + lv.smooth(g - lv.apply(x) if color else g, omega, ncp, color)
    return _ungrid(x, _nc(c), lv.np)


def _relaxation_value(c):
    """The reference's damping table (TPSS.h:121-163)."""
    if c.get("variant") == "multiplicative":
        return 1.0
    return 0.7 if c.get("patch") == "cell" else DAMPING[c["dim"]]


def _exact_step(c, seed):
    n = _n_dofs(c)
    x, b = _smooth(n, seed), _uniform(n, seed, 1)
    if c["distortion"]:
        mp = _Mapped(c["dim"], c["degree"], _nc(c), _coords(c, seed))
        return x + mp.smooth(b - mp.apply(x), 0.5 * DAMPING[c["dim"]])
    lv = _Level(c["dim"], c["degree"], _nc(c))
    x, b = _grid(x, _nc(c), lv.np), _grid(b, _nc(c), lv.np)
    return _ungrid(x + lv.smooth(b - lv.apply(x), DAMPING[c["dim"]]), _nc(c), lv.np)


def _exact_operator(c, seed):
    u = _smooth(_n_dofs(c), seed)
    if c["distortion"]:
        return _Mapped(c["dim"], c["degree"], _nc(c), _coords(c, seed)).apply(u)
    lv = _Level(c["dim"], c["degree"], _nc(c))
    return _ungrid(lv.apply(_grid(u, _nc(c), lv.np)), _nc(c), lv.np)


def _exact_transfer(c, seed):
    nc, np_ = _nc(c), c["degree"] + 1
    n = _n_dofs(c)
    nf, nfc = n * 2 ** c["dim"], [2 * m for m in _nc(c)]
    E = [_embed(c["degree"], m) for m in nc]
    fine = _smooth(nf, seed, 1) + _ungrid(_all_axes(E, _grid(_smooth(n, seed), nc, np_)), nfc, np_)
    coarse = _uniform(n, seed, 2) + _ungrid(_all_axes([e.T for e in E], _grid(_uniform(nf, seed, 3), nfc, np_)), nc, np_)
    return fine, coarse


def _exact_vcycle_case(c, seed):
    nc, np_ = [c["cells"]] * c["dim"], c["degree"] + 1
    g = _grid(_uniform(math.prod(nc) * np_ ** c["dim"], seed), nc, np_)
    return _ungrid(_exact_vcycle(c, g), nc, np_)


def _q_1d(k, nc):
    """1-D FE_Q mass, stiffness and C0IP bilaplacian matrices over all nodes of nc uniform cells."""
    z, h, gamma = _lobatto(k + 1), 1.0 / nc, k * (k + 1.0)
    qx, qw = _gauss(k + 1)
    V, D, E = _lagrange(z, qx)
    _, G, H = _lagrange(z, np.array([0.0, 1.0]))
    n = nc * k + 1
    M, L, B = np.zeros((n, n)), np.zeros((n, n)), np.zeros((n, n))
    for c in range(nc):
        s = slice(c * k, c * k + k + 1)
        M[s, s] += (V * qw) @ V.T * h
        L[s, s] += (D * qw) @ D.T / h
        B[s, s] += (E * qw) @ E.T / h ** 3
    for f in range(nc + 1):
        jump, mean = np.zeros(n), np.zeros(n)
        inner = 0 < f < nc
        if f > 0:
            jump[(f - 1) * k: f * k + 1] += G[:, 1] / h
            mean[(f - 1) * k: f * k + 1] += H[:, 1] / h ** 2 * (0.5 if inner else 1.0)
        if f < nc:
            jump[f * k: (f + 1) * k + 1] -= G[:, 0] / h
            mean[f * k: (f + 1) * k + 1] += H[:, 0] / h ** 2 * (0.5 if inner else 1.0)
        sigma = gamma / h if inner else 2 * gamma / h
        i = slice(max(0, (f - 1) * k), min(n, (f + 1) * k + 1))
        j, m = jump[i], mean[i]
        B[i, i] += sigma * np.outer(j, j) - np.outer(j, m) - np.outer(m, j)
    return M[1:-1, 1:-1], L[1:-1, 1:-1], B[1:-1, 1:-1]


def _exact_c0ip(c, seed):
    k, nc = c["degree"], c["cells"]
    M, L, B = _q_1d(k, nc)
    n, m = nc * k - 1, 2 * k - 1
    Mt, Lt, Bt = _dev(M), _dev(L), _dev(B)
    u, f = _smooth(n * n, seed).reshape(n, n), _uniform(n * n, seed, 1).reshape(n, n)
    Au = Mt @ u @ Bt.T + 2.0 * (Lt @ u @ Lt.T) + Bt @ u @ Mt.T
    w = f.unfold(0, m, k).unfold(1, m, k).contiguous()  # [vy, vx, m, m]
    P = nc - 1
    sub = [slice((v - 1) * k, (v - 1) * k + m) for v in range(1, nc)]
    if c["local"] == "fd":
        eig = [_gen_eig(M[s, s], B[s, s]) for s in (sub if P <= 3 else [sub[0], sub[1], sub[-1]])]
        at = list(range(P)) if P <= 3 else [0] + [1] * (P - 2) + [2]
        S, lam = _dev(np.array([eig[i][0] for i in at])), _dev(np.array([eig[i][1] for i in at]))
        w = torch.einsum("xij,yxaj->yxai", S.transpose(1, 2), w)
        w = torch.einsum("yij,yxja->yxia", S.transpose(1, 2), w)
        w = w / (lam[:, None, :, None] + lam[None, :, None, :])
        w = torch.einsum("xij,yxaj->yxai", S, w)
        w = torch.einsum("yij,yxja->yxia", S, w)
    else:
        at = list(range(P)) if P <= 3 else [0] + [1] * (P - 2) + [P - 1]
        x = torch.empty_like(w)
        for ky in sorted(set(at)):
            for kx in sorted(set(at)):
                sy, sx = sub[ky], sub[kx]
                K = np.kron(M[sy, sy], B[sx, sx]) + 2.0 * np.kron(L[sy, sy], L[sx, sx]) + np.kron(B[sy, sy], M[sx, sx])
                Ki = torch.linalg.inv(_dev(K))
                iy = torch.tensor([i for i, a in enumerate(at) if a == ky], device=DEV)
                ix = torch.tensor([i for i, a in enumerate(at) if a == kx], device=DEV)
                r = w[iy][:, ix].reshape(len(iy), len(ix), m * m)
                x[iy[:, None], ix[None, :]] = (r @ Ki.T).reshape(len(iy), len(ix), m, m)
        w = x
    out = torch.zeros_like(f)
    for a in range(m):
        for b in range(m):
            out[a: a + (P - 1) * k + 1: k, b: b + (P - 1) * k + 1: k] += w[:, :, a, b]
    return Au.reshape(-1), (DAMPING[2] * out).reshape(-1)


def _exact_mlp(c, seed):
    params, x, t = _mlp_data(c, seed)
    w, p, off = _widths(c), _dev(params), 0
    layers = []
    for a, b in zip(w[:-1], w[1:]):
        layers.append((p[off:off + a * b].reshape(b, a), p[off + a * b:off + a * b + b]))
        off += a * b + b
    acts = [x.to(F64)]
    for i, (W, b) in enumerate(layers):
        z = acts[-1] @ W.T + b
        acts.append(torch.tanh(z) if i + 1 < len(layers) else z)
    e = acts[-1] - t.to(F64)
    delta, grads = 2.0 * e / e.numel(), []
    for i in reversed(range(len(layers))):
        grads += [delta.sum(0), (delta.T @ acts[i]).reshape(-1)]
        if i:
            delta = (delta @ layers[i][0]) * (1.0 - acts[i] ** 2)
    return acts[-1], float((e * e).mean()), torch.cat(list(reversed(grads))).cpu().numpy()


_EXACT = dict(smoother=_exact_smoother, step=_exact_step, operator=_exact_operator, transfer=_exact_transfer,
              vcycle=_exact_vcycle_case, c0ip=_exact_c0ip, mlp=_exact_mlp)


def exact(case, seed):
    """None for the solve: where it stops within its tolerance has no value of its own."""
    return _EXACT[case["kind"]](case, seed) if case["kind"] in _EXACT else None
