"""The work this library is measured on: what a program does with it through
its public entry points, from a single plug-in call on a small level to the
whole assembly + solve of a two-million-dof problem.

A case is a dict of plain values; `kind` names what one pass does:

  plugin    the host-array kernels on one level (MatVect, Defect, SSOR,
            Prolongate, DefectRestriction): a host program that keeps its own
            iteration calls them one at a time, on small levels above all
  residual  one level's assembly from new coefficients, then its defect
            b - A x on device vectors: an outer (nonlinear, time or design)
            loop's residual evaluation
  vcycle    one preconditioner application z = MG(v) on device vectors
  solve     TSystemCD3D's Assemble + Solve: coefficients, assembly of every
            level, FGMRES to |r| <= 1e-10 |r0|, the solution to the host
  step      one Crank-Nicolson step of TSystemTCD3D: mass and stiffness on
            every level, the theta-scheme system, its solve, the restore
  train     the gradient of the stencil network on one problem's samples, as
            one rank of data-parallel training computes it

`coef` is the coefficient field (const, sine, lognormal, curl, rotating,
table), `prec` the V-cycle's precision, `smooth` its pre- and post-smoothing
steps (2 if not given), `mdml` the hierarchy with non-conforming levels.  The mesh of a case does not depend on the seed; the
coefficients, vectors, weights and samples do.
"""
import ctypes
import functools
import itertools
import math

import numpy as np
import torch

import parmoon_b200 as P
from parmoon_b200 import learned as PL
from parmoon_b200.configs import curl_modes, lognormal_modes

ELEMS = {"q1": P.Q1_HEX, "q2": P.Q2_HEX, "p2": P.P2_TET, "nq1": P.NQ1_HEX}
CELLS = {"q1": 1, "q2": 1, "p2": 6}  # cells per lattice cube
FORMS = {"const": P.FORM_SUPG, "curl": P.FORM_SUPG, "table": P.FORM_SUPG, "rotating": P.FORM_SUPG,
         "sine": P.FORM_GALERKIN, "lognormal": P.FORM_GALERKIN}
THETA_CN, TAU, T_OLD = (0.5, 0.5, 0.5, 0.5), 1e-3, 0.25
# V-cycles (= FGMRES iterations) of a solve to 1e-10, for the work estimate
CYCLES = {"const": 19, "sine": 6, "lognormal": 10, "curl": 15, "rotating": 10}


def listed():
    return [
        # a host program's own iteration on a small level: call latency
        dict(name="plugin_q1_16", kind="plugin", elem="q1", n=16),
        # residual of an ordinary Q2 SUPG level with an odd size (41^3 dofs)
        dict(name="residual_q2_20", kind="residual", elem="q2", n=20, coef="const"),
        # variable convection: coefficients and SUPG parameter at every quadrature point
        dict(name="residual_q1_curl_64", kind="residual", elem="q1", n=64, coef="curl"),
        # tetrahedra with a random diffusion field, 64 Fourier modes per point
        dict(name="residual_p2_lognormal_32", kind="residual", elem="p2", n=32, coef="lognormal"),
        # a host CoeffFct3D callback, tabulated and handed over before every assembly
        dict(name="residual_q1_table_32", kind="residual", elem="q1", n=32, coef="table"),
        # the preconditioner inside somebody else's Krylov method, FP64
        dict(name="vcycle_q2_32", kind="vcycle", elem="q2", n=32, levels=4, coef="const", prec="fp64"),
        # the smallest whole problem: Poisson on Q1 32^3
        dict(name="solve_q1_sine_32", kind="solve", elem="q1", n=32, levels=4, coef="sine", prec="fp32"),
        # the benchmark problem: convection-dominated SUPG on Q2 64^3
        dict(name="solve_q2_supg_64", kind="solve", elem="q2", n=64, levels=5, coef="const", prec="fp32"),
        # P2 tetrahedra with lognormal diffusion
        dict(name="solve_p2_lognormal_40", kind="solve", elem="p2", n=40, levels=4, coef="lognormal", prec="fp32"),
        # the non-conforming multilevel hierarchy, FP64 throughout
        dict(name="solve_mdml_q1_24", kind="solve", elem="q1", n=24, levels=4, coef="const", prec="fp64", mdml=True),
        # one time step of a rotating transport problem
        dict(name="step_q1_64", kind="step", elem="q1", n=64, levels=4, coef="rotating", prec="fp32"),
        # one rank's gradient of a training step on two samples at 64^3
        dict(name="train_q1_64", kind="train", elem="q1", n=64, samples=2, coef="curl"),
    ]


def _size(rng, coarse, most):
    """(cells per direction, levels): a coarse mesh refined 1 to 4 times, at most `most` cells."""
    sizes = [(c << k, k + 1) for c in coarse for k in range(1, 5) if 8 <= c << k <= most]
    target = math.exp(rng.uniform(math.log(8), math.log(most)))
    return rng.choice(sorted(sizes, key=lambda s: abs(math.log(s[0] / target)))[:6])


# coarsest meshes (cells per direction) whose active rows the dense coarsest solve takes
COARSE = {"q1": range(3, 10), "q2": (2, 3, 4, 5), "p2": (2, 3, 4, 5)}


def _n(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plugin", "residual", "residual", "vcycle", "solve", "solve", "step", "train"])
    if kind == "plugin":
        elem = rng.choice(["q1", "q2"])
        return dict(kind=kind, elem=elem, n=2 * _n(rng, 4, 24 if elem == "q1" else 12),
                    coef=rng.choice(["const", "sine", "curl"]))
    if kind == "residual":
        elem, coef, most = rng.choice([("q1", "const", 64), ("q2", "const", 32), ("q1", "curl", 64), ("q2", "curl", 24),
                                       ("p2", "lognormal", 32), ("q1", "table", 32), ("q2", "table", 16)])
        return dict(kind=kind, elem=elem, n=_n(rng, 8, most), coef=coef)
    if kind == "vcycle":
        elem = rng.choice(["q1", "q2"])
        n, levels = _size(rng, COARSE[elem], 32)
        return dict(kind=kind, elem=elem, n=n, levels=levels, coef=rng.choice(["const", "sine"]), prec="fp64",
                    smooth=rng.choice([1, 2, 3]))
    if kind == "solve":
        elem, coef, most = rng.choice([("q1", "sine", 48), ("q1", "const", 48), ("q2", "const", 40),
                                       ("p2", "lognormal", 40), ("q1", "curl", 48)])
        mdml = coef == "const" and rng.random() < 0.3
        n, levels = _size(rng, (3, 4, 5, 6) if mdml else COARSE[elem], min(most, 24) if mdml else most)
        case = dict(kind=kind, elem=elem, n=n, levels=levels + (1 if mdml else 0), coef=coef,
                    prec=rng.choice(["fp32", "fp32", "fp64"]), smooth=rng.choice([1, 2, 3]))
        return dict(case, mdml=True) if mdml else case
    if kind == "step":
        n, levels = _size(rng, COARSE["q1"], 64)
        return dict(kind=kind, elem="q1", n=n, levels=levels, coef="rotating", prec=rng.choice(["fp32", "fp64"]),
                    smooth=rng.choice([1, 2, 3]))
    return dict(kind=kind, elem="q1", n=_n(rng, 8, 64), samples=rng.choice([1, 2]), coef="curl")


# ------------------------------------------------------------------ inputs
def _levels_of(case):
    return case.get("levels", 2 if case["kind"] == "plugin" else 1)


@functools.lru_cache(maxsize=2)
def _hierarchy(elem, n, levels, mdml):
    if mdml:
        return P.mdml_hierarchy(ELEMS[elem], n, levels - 1)
    return P.struct_hierarchy(ELEMS[elem], n, levels, jitter=0.2 if elem == "p2" else 0.0, seed=1)


def _mesh(case):
    return _hierarchy(case["elem"], case["n"], _levels_of(case), bool(case.get("mdml")))


def _boundary(x, y, z):
    return (x < 1e-12).astype(float)


def _no_boundary(x, y, z):
    return np.zeros_like(x)


def _field(case, seed):
    """The seeded coefficient field as plain numbers (P.coeff's arguments)."""
    rng = np.random.default_rng([seed, 11])
    turn = rng.uniform(0.8, 1.25, 3)
    f = float(rng.uniform(0.5, 2.0))
    if case["coef"] == "sine":
        return dict(kind=P.COEF_SINE_RHS, eps=float(turn[0]))
    if case["coef"] == "lognormal":
        return dict(kind=P.COEF_LOGNORMAL, eps=1.0, f=f, modes=lognormal_modes(seed))
    if case["coef"] == "curl":
        modes, scale = curl_modes(seed, bmax=10.0)
        return dict(kind=P.COEF_CURL_FOURIER, eps=1e-3, b=(scale, 0.0, 0.0), f=f, modes=modes)
    if case["coef"] == "rotating":
        return dict(kind=P.COEF_ROTATING, eps=1e-4 * float(turn[0]), f=f)
    if case["coef"] == "table":
        return dict(kind=P.COEF_TABLE, eps=1e-3 * float(turn[0]), b=tuple(float(v) for v in turn), f=f)
    eps = 1e-3 if case.get("mdml") else 1e-6
    return dict(kind=P.COEF_CONST, eps=eps, b=(float(turn[0]), 0.5 * float(turn[1]), 0.25 * float(turn[2])), f=f)


def _table(field, xyz):
    """A host callback's values (eps, b, c, f) at the points xyz [..., 3]."""
    x, y, z = xyz[..., 0], xyz[..., 1], xyz[..., 2]
    b = field["b"]
    return np.stack([field["eps"] * (1.0 + x * y), b[0] * (1.0 + z), b[1] * (0.5 - x), b[2] * (1.0 + 0.5 * y),
                     0.1 + 0.0 * x, field["f"] * (1.0 + np.sin(3.0 * z))], axis=-1)


def _vector(seed, stream, n, na, scale=1.0):
    """A random level vector with smooth and rough parts, zero on the Dirichlet rows."""
    rng = np.random.default_rng([seed, stream])
    v = rng.standard_normal(n) + np.sin(np.arange(n) * (0.01 * rng.uniform(0.5, 2.0)))
    v[na:] = 0.0
    return scale * v


def _iterate_and_rhs(case, seed, F):
    """An iterate with its boundary values, and a right-hand side of the size of the matrix times it."""
    N, Na = F["N"], F["active_bound"]
    x, b = _vector(seed, 1, N, N), _vector(seed, 2, N, N, scale=case["n"] ** -2.0)
    b[Na:] = x[Na:]
    return x, b


def _params(case):
    kw = dict(precision=P.PREC_FP64 if case.get("prec") == "fp64" else P.PREC_FP32)
    kw["pre_smooth"] = kw["post_smooth"] = case.get("smooth", 2)
    if case["elem"] == "p2":
        kw["quad_rule"] = P.QUAD_KEAST5
    if case["kind"] == "solve" and case["elem"] == "q2":
        kw["restart"] = 40
    return P.default_params(**kw)


def _weights(seed):
    w = PL.init_weights(seed)
    return w + (0.01 * np.random.default_rng([seed, 5]).standard_normal(w.size)).astype(np.float32)


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def prepare(case, seed):
    levels, kind = _mesh(case), case["kind"]
    F, top = levels[-1], len(levels) - 1
    N, Na = F["N"], F["active_bound"]
    field = _field(dict(case, coef=case.get("coef", "const")), seed)
    h = P.Handle(len(levels), _params(case))
    P.load_hierarchy(h, levels, dirichlet=_no_boundary if kind in ("step", "train") else _boundary)
    s = dict(kind=kind, h=h, top=top, form=FORMS[case.get("coef", "const")])
    if kind != "step":
        s["coef"] = P.coeff(**field)
        h.set_coefficients(s["coef"])
    if kind == "plugin":
        h.assemble(-1, s["form"], copy_out=False)
        s["x"], s["b"] = _iterate_and_rhs(case, seed, F)
        s["c"] = _vector(seed, 3, levels[0]["N"], levels[0]["N"])
    elif kind == "residual":
        s["x"], s["b"] = (torch.from_numpy(v).cuda() for v in _iterate_and_rhs(case, seed, F))
        s["r"], s["norm"] = torch.empty_like(s["x"]), torch.empty(1, dtype=torch.float64, device="cuda")
        if case["coef"] == "table":
            s["table"] = _table(field, h.quad_points(top))
    elif kind == "vcycle":
        h.assemble(-1, s["form"], copy_out=False)
        s["v"] = torch.from_numpy(_vector(seed, 1, N, Na)).cuda()
        s["z"] = torch.empty_like(s["v"])
    elif kind == "solve":
        s["out"] = torch.empty(N, dtype=torch.float64).pin_memory().numpy()
    elif kind == "step":
        s["u"] = _bump(F, seed)
        s["coefs"] = [P.coeff(t=t, **field) for t in (T_OLD, T_OLD + TAU)]
        s["out"] = torch.empty(N, dtype=torch.float64).pin_memory().numpy()
    else:
        h.set_lattice(0, case["n"] + 1, F["dof_lat"])
        h.assemble(-1, s["form"], copy_out=False)
        h.set_learned_weights(_weights(seed))
        e = [_vector(seed, k, N, Na) for k in range(case["samples"])]
        e = [v / np.linalg.norm(v) for v in e]
        r = [h.matvec(0, v) for v in e]
        for v in r:
            v[Na:] = 0.0
        s["E"], s["R"] = (torch.from_numpy(np.stack(v)).cuda() for v in (e, r))
    torch.cuda.synchronize()
    return s


def _bump(F, seed):
    """A Gaussian bump, the transported quantity of a time step."""
    x = F["dof_xyz"] - np.random.default_rng([seed, 3]).uniform(0.3, 0.7, 3)
    u = np.exp(-(x ** 2).sum(1) / (2 * 0.05 ** 2))
    u[F["active_bound"]:] = 0.0
    return u


def run(s):
    h, kind, top = s["h"], s["kind"], s["top"]
    if kind == "plugin":
        y = h.matvec(top, s["x"])
        r, norm = h.defect(top, s["x"], s["b"])
        return dict(y=y, r=r, norm=norm, sol=h.ssor(top, s["b"], s["x"]), fine=h.prolongate(top, s["c"]),
                    coarse=h.restrict(top, s["x"]))
    if kind == "residual":
        if "table" in s:
            h.set_coefficient_table(top, s["table"])
        h.set_coefficients(s["coef"])
        h.assemble(top, s["form"], copy_out=False)
        P._check(P.lib().pmg_defect_noalloc(h.h, ctypes.c_int(top), _ptr(s["x"]), _ptr(s["b"]), _ptr(s["r"]),
                                            _ptr(s["norm"])))
        return dict(r=s["r"], norm=s["norm"])
    if kind == "vcycle":
        h.vcycle(s["v"].data_ptr(), s["z"].data_ptr())
        return s["z"]
    if kind == "solve":
        h.set_coefficients(s["coef"])
        h.assemble(-1, s["form"], copy_out=False)
        h.solve()
        return h.get_solution(out=s["out"])
    if kind == "step":
        h.set_coefficients(s["coefs"][0])
        h.assemble(-1, P.FORM_MASS_SUPG, copy_out=False)
        h.set_coefficients(s["coefs"][1])
        h.assemble(-1, P.FORM_SUPG, copy_out=False)
        B = h.tcd_system(TAU, THETA_CN, u_old=s["u"])
        h.solve()
        h.tcd_restore()
        return dict(B=B, u=h.get_solution(out=s["out"]))
    loss, grad = h.learned_train_step(top, s["E"].data_ptr(), s["R"].data_ptr(), s["E"].shape[0], 0.0, want_grad=True)
    return dict(loss=loss, grad=grad)


# ------------------------------------------------------------------ work
def work(case):
    """Bytes and operations of one pass.  A matrix entry costs 8 bytes of value
    and 2 of column (4 + 2 in an FP32 V-cycle); an assembly writes the matrix
    and reads the mesh; an SSOR step needs every entry once (the lower part
    forward, the upper part backward), so a V-cycle with two pre- and two
    post-smoothing steps and a defect reads the matrix five times; coarser
    levels add a seventh.  A solve does that once per iteration, with one FP64
    product."""
    n, elem, kind = case["n"], case["elem"], case["kind"]
    p = 1 if elem == "q1" else 2
    nloc, cells = {"q1": 8, "q2": 27, "p2": 10}[elem], n ** 3 * CELLS[elem]
    rows = (p * n + 1) ** 3
    nnz = rows * {"q1": 27, "q2": 64, "p2": 28}[elem]
    val = 6 if case.get("prec") == "fp32" else 10
    assemble = dict(bytes=cells * (4 * nloc + 96) + 8 * nnz, flops=cells * 32 * nloc ** 2)
    product = dict(bytes=10 * nnz + 24 * rows, flops=2 * nnz)
    reads = 2 * case.get("smooth", 2) + 1
    cycle = dict(bytes=reads * val * nnz * 8 / 7, flops=(4 * reads - 2) * nnz * 8 / 7)

    def total(*parts):
        return {k: float(sum(m * d[k] for m, d in parts)) for k in ("bytes", "flops")}

    if kind == "plugin":
        return total((4, product))
    if kind == "residual":
        return total((1, assemble), (1, product))
    if kind == "vcycle":
        return total((1, cycle))
    if kind == "solve":
        its = CYCLES[case["coef"]]
        return total((8 / 7, assemble), (its, cycle), (its, product))
    if kind == "step":
        its = CYCLES[case["coef"]]
        return total((16 / 7, assemble), (its, cycle), (its + 2, product))
    net = 2 * 27 * (27 * 32 + 32 * 32 + 32 * 27) * rows
    m = case["samples"]
    return dict(bytes=float((1 + 2 * m) * 10 * nnz + 16 * rows * m), flops=float(net * (1 + 2 * m)))


# ------------------------------------------------------------------ exact values
# Plain torch in FP64: local matrices from monomial bases, sparse level
# matrices, a colour-by-colour V-cycle and GMRES with it.
def _cuda(a, dtype=torch.float64):
    return torch.as_tensor(np.asarray(a)).to("cuda", dtype)


def _quadrature(elem):
    if elem == P.P2_TET:  # 5 points, degree 3
        a, b = 1 / 6, 1 / 2
        pts = [(.25, .25, .25), (a, a, a), (a, a, b), (a, b, a), (b, a, a)]
        return np.array(pts), np.array([-2 / 15] + [3 / 40] * 4)
    x, w = np.polynomial.legendre.leggauss(2 if elem == P.Q1_HEX else 3)
    m = len(x)
    pts = np.array([(x[k], x[j], x[i]) for i in range(m) for j in range(m) for k in range(m)])
    wts = np.array([w[k] * w[j] * w[i] for i in range(m) for j in range(m) for k in range(m)])
    return pts, wts


def _monomials(elem, X):
    """Values and gradients [points, functions, 4] (d/dx, d/dy, d/dz, value) of the element's polynomial space."""
    if elem == P.NQ1_HEX:
        terms = [[(1., (0, 0, 0))], [(1., (1, 0, 0))], [(1., (0, 1, 0))], [(1., (0, 0, 1))],
                 [(1., (2, 0, 0)), (-1., (0, 2, 0))], [(1., (2, 0, 0)), (-1., (0, 0, 2))]]
    elif elem == P.P2_TET:
        terms = [[(1., e)] for e in itertools.product(range(3), repeat=3) if sum(e) <= 2]
    else:
        terms = [[(1., e)] for e in itertools.product(range(2 if elem == P.Q1_HEX else 3), repeat=3)]
    out = np.zeros((len(X), len(terms), 4))
    for m, term in enumerate(terms):
        for c, e in term:
            powers = [X[:, d] ** e[d] for d in range(3)]
            slopes = [e[d] * X[:, d] ** max(e[d] - 1, 0) for d in range(3)]
            out[:, m, 3] += c * powers[0] * powers[1] * powers[2]
            for d in range(3):
                out[:, m, d] += c * slopes[d] * powers[(d + 1) % 3] * powers[(d + 2) % 3]
    return out


def _maps(L):
    """Affine maps x = x0 + J xi of the cells, from [-1,1]^3 or the unit simplex."""
    v = _cuda(L["cell_vert"]).reshape(-1, 8, 3)
    if L["elem"] == P.P2_TET:
        return v[:, 0], torch.stack([v[:, k] - v[:, 0] for k in (1, 2, 3)], dim=2), v
    J = torch.stack([(v[:, k] - v[:, 0]) / 2 for k in (1, 3, 4)], dim=2)
    return v[:, 0] + J.sum(2), J, v


def _coefficients(field, t, X):
    """eps, b, c, f at the points X [cells, points, 3]."""
    x, y, z = X[..., 0], X[..., 1], X[..., 2]
    one = torch.ones_like(x)
    eps, f = field["eps"] * one, field.get("f", 1.0) * one
    b = torch.stack([v * one for v in field.get("b", (0.0, 0.0, 0.0))], dim=-1)
    if field["kind"] == P.COEF_TABLE:
        tab = _cuda(_table(field, X.cpu().numpy()))
        return tab[..., 0], tab[..., 1:4], tab[..., 4], tab[..., 5]
    if field["kind"] == P.COEF_SINE_RHS:
        f = 3 * math.pi ** 2 * eps * torch.sin(math.pi * x) * torch.sin(math.pi * y) * torch.sin(math.pi * z)
    elif field["kind"] == P.COEF_LOGNORMAL:
        g = torch.zeros_like(x)
        for m in field["modes"]:
            g += m[3] * torch.cos(2 * math.pi * (m[0] * x + m[1] * y + m[2] * z) + m[4])
        eps = eps * torch.exp(g)
    elif field["kind"] == P.COEF_CURL_FOURIER:
        curl = torch.zeros_like(X)
        for m in field["modes"]:
            s = -2 * math.pi * m[3] * torch.sin(2 * math.pi * (m[0] * x + m[1] * y + m[2] * z) + m[4])
            curl += s[..., None] * _cuda(np.cross(m[0:3], m[5:8]))
        b = field["b"][0] * curl
    elif field["kind"] == P.COEF_ROTATING:
        b = torch.stack([0.5 - y, x - 0.5, 0.2 * math.sin(2 * math.pi * t) * one], dim=-1)
    return eps, b, 0 * one, f


def _local(L, field, form, t=0.0):
    """Local matrices [cells, nloc, nloc] (test, trial) and right-hand sides of one form."""
    elem, nloc = L["elem"], P.NLOC[L["elem"]]
    pts, wts = _quadrature(elem)
    x0, J, vert = _maps(L)
    Ji = torch.linalg.inv(J)
    nodes = _cuda(L["dof_xyz"])[torch.as_tensor(L["elem_dof"][:nloc], dtype=torch.long, device="cuda")]
    ref = torch.round(2 * (nodes - x0[0]) @ Ji[0].T).cpu().numpy() / 2
    U = _cuda(np.einsum("qma,ml->qla", _monomials(elem, pts), np.linalg.inv(_monomials(elem, ref)[:, :, 3])))
    X = x0[:, None] + torch.einsum("cde,qe->cqd", J, _cuda(pts))
    eps, b, c, f = _coefficients(field, t, X)
    K = Ji @ Ji.transpose(1, 2)
    bh = torch.einsum("cpd,cqd->cqp", Ji, b)
    supg = form in (P.FORM_SUPG, P.FORM_MASS_SUPG)
    delta = torch.zeros_like(eps)
    if supg:
        size = (vert.amax(1) - vert.amin(1))
        s = b[:, 0] / size
        den = 0.5 * sum((s[:, 0] + i * s[:, 1] + k * s[:, 2]).abs() for i in (1, -1) for k in (1, -1))
        nb = b.norm(dim=2)
        hk = (2 * b[:, 0].norm(dim=1) / den)[:, None]
        nu = 0.5 if elem == P.Q2_HEX else 1.0
        a = nu * nb * hk / (2 * eps)
        delta = nu * hk * (1 / torch.tanh(a) - 1 / a) / (2 * nb)
    D = torch.zeros(*eps.shape, 4, 4, dtype=torch.float64, device="cuda")
    if form in (P.FORM_MASS, P.FORM_MASS_SUPG):
        D[..., 3, 3] = 1.0
        D[..., :3, 3] = delta[..., None] * bh
    else:
        D[..., :3, :3] = eps[..., None, None] * K[:, None] + delta[..., None, None] * bh[..., None] * bh[..., None, :]
        D[..., 3, :3] = bh
        D[..., 3, 3] = c
        D[..., :3, 3] = (delta * c)[..., None] * bh
    w = _cuda(wts) * torch.linalg.det(J).abs()[:, None]
    tab = torch.einsum("qia,qjb->qabij", U, U).reshape(-1, nloc * nloc)
    A = torch.cat([(w[k][..., None, None] * D[k]).flatten(1) @ tab for k in torch.split(
        torch.arange(len(w), device="cuda"), 65536)]).reshape(-1, nloc, nloc)
    test = torch.cat([delta[..., None] * bh, torch.ones_like(w)[..., None]], dim=2)
    return A, torch.einsum("cq,cqa,qla->cl", w * f, test, U)


def _system(L, A, f, boundary):
    """Sparse level matrix with identity Dirichlet rows, and its right-hand side."""
    N, Na, nloc = L["N"], L["active_bound"], P.NLOC[L["elem"]]
    dof = torch.as_tensor(L["elem_dof"], dtype=torch.long, device="cuda").reshape(-1, nloc)
    row, col = dof[:, :, None].expand_as(A).reshape(-1), dof[:, None, :].expand_as(A).reshape(-1)
    keep = row < Na
    d = torch.arange(Na, N, device="cuda")
    idx = torch.stack([torch.cat([row[keep], d]), torch.cat([col[keep], d])])
    val = torch.cat([A.reshape(-1)[keep], torch.ones(N - Na, dtype=torch.float64, device="cuda")])
    M = torch.sparse_coo_tensor(idx, val, (N, N)).coalesce().to_sparse_csr()
    rhs = torch.zeros(N, dtype=torch.float64, device="cuda").index_add_(0, dof.reshape(-1), f.reshape(-1))
    xyz = np.asarray(L["dof_xyz"])[Na:]
    rhs[Na:] = _cuda(boundary(xyz[:, 0], xyz[:, 1], xyz[:, 2]))
    return M, rhs


def _rows(M, rows):
    """The given rows of a CSR matrix."""
    rp, col, val = M.crow_indices(), M.col_indices(), M.values()
    n = rp[rows + 1] - rp[rows]
    out = torch.cat([torch.zeros(1, dtype=torch.long, device="cuda"), n.cumsum(0)])
    at = torch.arange(int(out[-1]), device="cuda") + torch.repeat_interleave(rp[rows] - out[:-1], n)
    return torch.sparse_csr_tensor(out, col[at], val[at], (len(rows), M.shape[1]))


class _Level:
    def __init__(self, L, M, n_coarse):
        self.M, self.Na, self.N = M, L["active_bound"], L["N"]
        rp, col, val = M.crow_indices(), M.col_indices(), M.values()
        row = torch.repeat_interleave(torch.arange(self.N, device="cuda"), rp[1:] - rp[:-1])
        self.diag = torch.zeros(self.N, dtype=torch.float64, device="cuda")
        self.diag[row[row == col]] = val[row == col]
        self.colors = None
        if L.get("colors") is not None:
            c = torch.as_tensor(L["colors"][:self.Na], device="cuda")
            self.colors = [(r, _rows(M, r)) for r in (torch.nonzero(c == k)[:, 0] for k in range(L["n_colors"])) if len(r)]
        if n_coarse:
            rp, col, val = L["P"]
            at = torch.as_tensor(np.stack([np.repeat(np.arange(self.N), np.diff(rp)), col]), device="cuda")
            self.P = torch.sparse_coo_tensor(at, _cuda(val), (self.N, n_coarse)).coalesce().to_sparse_csr()
            self.R = torch.sparse_coo_tensor(at.flip(0), _cuda(val), (n_coarse, self.N)).coalesce().to_sparse_csr()

    def smooth(self, x, f, steps):
        x[self.Na:] = f[self.Na:]
        for _ in range(steps):
            if self.colors is None:  # damped Jacobi, as a preconditioner only
                x[:self.Na] += 0.6 * ((f - self.M @ x) / self.diag)[:self.Na]
                continue
            for r, A in self.colors + self.colors[::-1]:
                x[r] += (f[r] - A @ x) / self.diag[r]


def _hierarchy_exact(levels, mats):
    sizes = [0] + [L["N"] for L in levels]
    out = [_Level(L, M, n) for L, M, n in zip(levels, mats, sizes)]
    out[0].dense = torch.linalg.lu_factor(out[0].M.to_dense())
    return out


def _vcycle(lv, k, f, steps=2):
    L = lv[k]
    if k == 0:
        return torch.linalg.lu_solve(*L.dense, f[:, None])[:, 0]
    x = torch.zeros_like(f)
    L.smooth(x, f, steps)
    fc = L.R @ (f - L.M @ x)
    fc[lv[k - 1].Na:] = 0
    x[:L.Na] += (L.P @ _vcycle(lv, k - 1, fc, steps))[:L.Na]
    L.smooth(x, f, steps)
    return x


def _gmres(lv, b, restarts=6, m=40):
    M, top = lv[-1].M, len(lv) - 1
    x = torch.zeros_like(b)
    x[lv[-1].Na:] = b[lv[-1].Na:]
    r0 = None
    for _ in range(restarts):
        r = b - M @ x
        beta = float(r.norm())
        r0 = beta if r0 is None else r0
        if beta <= 2e-15 * r0:
            break
        V, Z, H = [r / beta], [], np.zeros((m + 1, m))
        for j in range(m):
            Z.append(_vcycle(lv, top, V[j]))
            w = M @ Z[j]
            for i in list(range(j + 1)) * 2:
                c = float(w @ V[i])
                H[i, j] += c
                w = w - c * V[i]
            H[j + 1, j] = float(w.norm())
            e1 = np.zeros(j + 2)
            e1[0] = beta
            y = np.linalg.lstsq(H[:j + 2, :j + 1], e1, rcond=None)[0]
            if H[j + 1, j] <= 1e-300 or np.linalg.norm(e1 - H[:j + 2, :j + 1] @ y) <= 1e-15 * r0:
                break
            V.append(w / H[j + 1, j])
        x = x + sum(float(c) * z for c, z in zip(y, Z))
    return x


def _exact_gradient(case, seed, L, M):
    """Loss and gradient of the stencil network; weights and every layer's input are rounded to BF16, as the network
    is defined, everything else is FP64."""
    n1, N, Na = case["n"] + 1, L["N"], L["active_bound"]

    def rounded(x):
        return x + (x.to(torch.bfloat16).double() - x).detach()

    lat = torch.as_tensor(L["dof_lat"], dtype=torch.long, device="cuda")
    rp, col, val = M.crow_indices(), M.col_indices(), M.values()
    row = torch.repeat_interleave(torch.arange(N, device="cuda"), rp[1:] - rp[:-1])
    act = row < Na
    row, col, val = row[act], col[act], val[act]
    diag = torch.ones(N, dtype=torch.float64, device="cuda")
    diag[row[row == col]] = val[row == col]
    a, c = lat[row], lat[col]
    k = sum(3 ** d * ((c // n1 ** d) % n1 - (a // n1 ** d) % n1 + 1) for d in range(3))
    x = torch.zeros(n1 ** 3, 27, dtype=torch.float64, device="cuda")
    x[a, k] = (val / diag[row]).float().to(torch.bfloat16).double()
    scale = torch.zeros(n1 ** 3, dtype=torch.float64, device="cuda")
    scale[lat[:Na]] = 1 / diag[:Na]

    def shift(v, o):
        """v at the neighbour with offset number o, zero outside the lattice."""
        g = torch.nn.functional.pad(v.T.reshape(-1, n1, n1, n1), (1,) * 6)
        i, j, m = o % 3, o // 3 % 3, o // 9
        return g[:, m:m + n1, j:j + n1, i:i + n1].reshape(len(g), -1).T

    w = _cuda(_weights(seed)).to(torch.bfloat16).double().requires_grad_()
    at = 0
    for co, ci in ((32, 27), (32, 32), (27, 32)):
        W, bias = w[at:at + co * ci * 27].reshape(co, ci, 27), w[at + co * ci * 27:at + co * ci * 27 + co]
        at += co * ci * 27 + co
        x = sum(shift(x, o) @ W[:, :, o].T for o in range(27)) + bias
        if co != 27:
            x = rounded(torch.relu(x))
    stencil = x * scale[:, None]
    loss = 0
    for s in range(case["samples"]):
        e = _vector(seed, s, N, Na)
        e = _cuda(e / np.linalg.norm(e))
        r = M @ e
        r[Na:] = 0
        grid = torch.zeros(n1 ** 3, 1, dtype=torch.float64, device="cuda")
        grid[lat, 0] = r
        corr = sum(stencil[:, o] * shift(grid, o)[:, 0] for o in range(27))
        u = e.clone()
        u[:Na] = e[:Na] - corr[lat[:Na]]
        v = _Product.apply(M, u)
        loss = loss + (v @ v) / (r @ r) / case["samples"]
    loss.backward()
    return dict(loss=float(loss.detach()), grad=w.grad)


class _Product(torch.autograd.Function):
    """M @ u with the gradient M^T g."""

    @staticmethod
    def forward(ctx, M, u):
        ctx.M = M
        return M @ u

    @staticmethod
    def backward(ctx, g):
        M = ctx.M
        row = torch.repeat_interleave(torch.arange(M.shape[0], device="cuda"), M.crow_indices()[1:] - M.crow_indices()[:-1])
        return None, torch.zeros_like(g).index_add_(0, M.col_indices(), M.values() * g[row])


def exact(case, seed):
    levels, kind = _mesh(case), case["kind"]
    F = levels[-1]
    field = _field(dict(case, coef=case.get("coef", "const")), seed)
    form = FORMS[case.get("coef", "const")]
    if kind == "residual":
        A, _ = _local(F, field, form)
        x, b = (_cuda(v) for v in _iterate_and_rhs(case, seed, F))
        dof = torch.as_tensor(F["elem_dof"], dtype=torch.long, device="cuda").reshape(A.shape[:2])
        y = torch.zeros_like(x).index_add_(0, dof.reshape(-1), torch.einsum("cij,cj->ci", A, x[dof]).reshape(-1))
        y[F["active_bound"]:] = x[F["active_bound"]:]
        return dict(r=b - y, norm=(b - y).norm().reshape(1))
    boundary = _no_boundary if kind in ("step", "train") else _boundary
    if kind == "train":
        return _exact_gradient(case, seed, F, _system(F, *_local(F, field, form), boundary)[0])
    if kind == "step":
        mats, sides = [], []
        for L in levels:
            M, f0 = _system(L, *_local(L, field, P.FORM_MASS_SUPG, T_OLD), boundary)
            A, f1 = _system(L, *_local(L, field, form, T_OLD + TAU), boundary)
            u, na = _cuda(_bump(F, seed)), L["active_bound"]
            if L is F:
                rhs = TAU * 0.5 * (f0 + f1) + M @ u - TAU * 0.5 * (A @ u)
                rhs[na:] = f1[na:]
            inside = torch.repeat_interleave(torch.arange(L["N"], device="cuda") < na,
                                             M.crow_indices()[1:] - M.crow_indices()[:-1])
            mats.append(torch.sparse_csr_tensor(M.crow_indices(), M.col_indices(), torch.where(
                inside, M.values() + TAU * 0.5 * A.values(), M.values()), M.shape))
        return dict(B=rhs, u=_gmres(_hierarchy_exact(levels, mats), rhs))
    pairs = [_system(L, *_local(L, field, form), boundary) for L in levels]
    lv = _hierarchy_exact(levels, [M for M, _ in pairs])
    if kind == "solve":
        return _gmres(lv, pairs[-1][1])
    if kind == "vcycle":
        return _vcycle(lv, len(lv) - 1, _cuda(_vector(seed, 1, F["N"], F["active_bound"])), case.get("smooth", 2))
    T = lv[-1]
    x, b = (_cuda(v) for v in _iterate_and_rhs(case, seed, F))
    c = _cuda(_vector(seed, 3, lv[0].N, lv[0].N))
    r, sol = b - T.M @ x, x.clone()
    T.smooth(sol, b, 1)
    return dict(y=T.M @ x, r=r, norm=float(r.norm()), sol=sol, fine=T.P @ c, coarse=T.R @ x)
