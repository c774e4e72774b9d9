"""Workloads of the Stokes path: what they run, on which inputs, and what they have to give.

A case is a dict of plain values. `listed()` names the standing ones, `draw(rng)` makes more of the same ranges,
`prepare(case, seed)` builds what a program holds before the call (mesh hierarchy, coefficient, operator or solver,
vectors), `run(state)` makes one pass through the public entry points of `terra_b200`, `work(case)` counts the bytes
and operations the pass needs at least, `tolerance(case)` states how far another correct implementation may be off and
`exact(case, seed)` gives the results of the operators in 64 bits from a plain torch restatement of the discretisation.

Kinds of case (`op`):

* `apply`       one epsilon-div-div operator apply: the unit of work of every smoother and residual;
* `stokes`      one Stokes block apply [A B^T; B 0]: the outer residual and Krylov operator;
* `vjp`         the backward pass of the apply: gradient in the per-cell log-viscosity, and A^T lambda;
* `galerkin`    one apply of a stored Galerkin operator one level below: the coarse smoothers' unit of work;
* `gca_build`   Galerkin operators of the next two levels and one apply of each: the set-up after a change of viscosity;
* `precondition` one block-triangular preconditioner application (Schur step, B^T, one V-cycle);
* `cg`          a velocity solve by multigrid-preconditioned conjugate gradients;
* `solve`       a Stokes solve by FGMRES to 1e-8.

Levels: a level l has 10 diamonds of (2^l + 1)^2 node columns; the radial level may differ from the lateral one.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = next(p for p in (os.path.join(os.path.abspath(r or "."), "terra-ng_b200") for r in ["."] + sys.path)
            if os.path.isdir(p))
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import terra_b200 as T  # noqa: E402

R_MIN, R_MAX = 0.55, 1.0
NEUMANN, DIRICHLET, FREESLIP = 0, 1, 2


# ----------------------------------------------------------------------------------------------------------------
# Cases
# ----------------------------------------------------------------------------------------------------------------
def _case(op, lat, rad=None, dtype="f64", bcs=(DIRICHLET, FREESLIP), q0=False, **kw):
    c = {"op": op, "lat": lat, "rad": lat if rad is None else rad, "dtype": dtype, "cmb": bcs[0], "surface": bcs[1],
         "q0": q0}
    c.update(kw)
    return c


def listed():
    out = [
        # a small apply, where latency and launches count: the coarse levels of a hierarchy, and a regional test mesh
        ("apply_f64_L3", _case("apply", 3, bcs=(DIRICHLET, DIRICHLET))),
        # the smoother's operator of the mixed-precision level-6 solve, by far the most frequent call
        ("apply_f32_L6", _case("apply", 6, dtype="f32")),
        # the same operator in FP64: the outer residual and the FP64 V-cycle
        ("apply_f64_L6", _case("apply", 6)),
        # a shell that is finer laterally than radially, free-slip on both sides, per-cell viscosity
        ("apply_f32_lat6_rad5_cells", _case("apply", 6, 5, dtype="f32", bcs=(FREESLIP, FREESLIP), q0=True)),
        # the largest mesh one program keeps on the device: 21.5 million nodes, per-cell viscosity
        ("apply_f64_L7_cells", _case("apply", 7, q0=True)),
        # the Krylov operator of the Stokes solve
        ("stokes_f64_L6", _case("stokes", 6)),
        # the backward pass of the adjoint viscosity inversion
        ("vjp_f64_L5_cells", _case("vjp", 5, q0=True)),
        # the level-5 coarse operator of a level-6 hierarchy
        ("galerkin_f64_L5", _case("galerkin", 6)),
        # a time step with a new viscosity rebuilds the coarse operators
        ("gca_build_L6", _case("gca_build", 6)),
        # the preconditioner, FP32 V-cycle: the body of every FGMRES iteration
        ("precondition_mixed_L6", _case("precondition", 6, dtype="f32", levels=5)),
        # a velocity solve in FP64 on a mesh of moderate size: many short kernels
        ("cg_f64_L4", _case("cg", 4, bcs=(DIRICHLET, DIRICHLET), levels=3)),
        # the whole mixed-precision solve of a mantle-convection time step
        ("solve_mixed_L6", _case("solve", 6, dtype="f32", levels=5)),
    ]
    return [dict(c, name=n) for n, c in out]


def draw(rng):
    op = rng.choice(["apply"] * 4 + ["stokes", "vjp", "galerkin", "gca_build", "precondition", "cg", "solve"])
    bcs = rng.choice([(DIRICHLET, FREESLIP), (DIRICHLET, DIRICHLET), (FREESLIP, DIRICHLET), (NEUMANN, NEUMANN),
                      (FREESLIP, FREESLIP), (NEUMANN, DIRICHLET)])
    pinned = rng.choice([(DIRICHLET, FREESLIP), (DIRICHLET, DIRICHLET)])
    dtype = rng.choice(["f32", "f64"])
    q0 = rng.random() < 0.4
    if op == "apply":
        lat = rng.randint(2, 7)
        rad = min(7, max(1, lat + rng.randint(-2, 1)))
        return _case(op, lat, rad, dtype, bcs, q0)
    if op == "stokes":
        lat = rng.randint(2, 6)
        return _case(op, lat, max(2, lat + rng.choice([-1, 0])), dtype, bcs, q0)
    if op == "vjp":
        lat = rng.randint(2, 6)
        return _case(op, lat, max(1, lat + rng.choice([-1, 0])), dtype, bcs, True)
    if op == "galerkin":
        lat = rng.randint(3, 6)
        return _case(op, lat, max(2, lat + rng.choice([-1, 0])), "f64", bcs, q0)
    if op == "gca_build":
        lat = rng.randint(3, 6)
        return _case(op, lat, max(3, lat + rng.choice([-1, 0])), "f64", bcs, q0)
    if op == "precondition":
        lat = rng.randint(4, 6)
        return _case(op, lat, lat - rng.randint(0, 1), dtype, pinned, False, levels=lat - 1)
    if op == "cg":
        lat = rng.randint(3, 5)
        return _case(op, lat, lat, dtype, pinned, False, levels=lat - 1)
    lat = rng.randint(3, 5)
    return _case(op, lat, lat, dtype, pinned, False, levels=lat - 1)


# ----------------------------------------------------------------------------------------------------------------
# Mesh in plain numpy (the ten icosahedral diamonds, refined by normalised midpoints)
# ----------------------------------------------------------------------------------------------------------------
_DIAMONDS = [(0, 5, 6, 1), (0, 1, 7, 2), (0, 2, 8, 3), (0, 3, 9, 4), (0, 4, 10, 5),
             (11, 7, 1, 6), (11, 8, 2, 7), (11, 9, 3, 8), (11, 10, 4, 9), (11, 6, 5, 10)]


def _unit(v):
    return v / np.sqrt((v * v).sum(-1, keepdims=True))


def _sphere(lat):
    """(10, n, n, 3) unit vectors of the node columns."""
    fifth = 0.4 * math.asin(1.0)
    w = 2.0 * math.acos(1.0 / (2.0 * math.sin(fifth)))
    base = np.zeros((12, 3))
    base[0], base[11] = (0, 0, 1), (0, 0, -1)
    for k in range(1, 6):
        a, b = 2.0 * (k - 0.5) * fifth, 2.0 * (k - 1) * fifth
        base[k] = (math.sin(w) * math.cos(a), math.sin(w) * math.sin(a), math.cos(w))
        base[k + 5] = (math.sin(w) * math.cos(b), math.sin(w) * math.sin(b), -math.cos(w))
    c = np.zeros((10, 2, 2, 3))
    for d, m in enumerate(_DIAMONDS):
        left, right = (1, 3) if d < 5 else (3, 1)
        c[d, 0, 0], c[d, 1, 0], c[d, 1, 1], c[d, 0, 1] = base[m[0]], base[m[left]], base[m[2]], base[m[right]]
    for _ in range(lat):
        n = c.shape[1]
        f = np.zeros((10, 2 * n - 1, 2 * n - 1, 3))
        f[:, ::2, ::2] = c
        f[:, 1::2, ::2] = _unit(c[:, :-1] + c[:, 1:])
        f[:, ::2, 1::2] = _unit(c[:, :, :-1] + c[:, :, 1:])
        f[:, 1::2, 1::2] = _unit(c[:, 1:, :-1] + c[:, :-1, 1:])
        c = f
    return c


def _radii(rad):
    return np.linspace(R_MIN, R_MAX, (1 << rad) + 1)


def _unique_columns(n):
    """For every stored column the index of its geometric point (copies on diamond edges share it)."""
    key = np.round(_sphere(n).reshape(-1, 3) * 1e7).astype(np.int64)
    _, inv = np.unique(key, axis=0, return_inverse=True)
    return torch.tensor(inv.reshape(-1), device="cuda")


# ----------------------------------------------------------------------------------------------------------------
# Inputs: fields that are functions of the position, so copies of a node agree
# ----------------------------------------------------------------------------------------------------------------
def _dtype(case):
    return torch.float32 if case["dtype"] == "f32" else torch.float64


def _waves(points, radii, rng, kmax, terms=6):
    """Sum of `terms` plane waves, wave numbers log-uniform in [1, kmax]; points (..., 3) unit vectors, times radii."""
    out = 0.0
    p = torch.tensor(points, device="cuda")
    r = torch.tensor(radii, device="cuda")
    for _ in range(terms):
        k = rng.standard_normal(3)
        k *= math.exp(rng.uniform(0.0, math.log(kmax))) / np.linalg.norm(k)
        ph = rng.uniform(0.0, 2.0 * math.pi)
        lat = p @ torch.tensor(k, device="cuda")
        out = out + rng.standard_normal() * torch.sin(lat[..., None] * r + ph)
    return out


def _velocity(lat, rad, rng):
    """Smooth and grid-scale parts, as the vectors a smoother and a Krylov method apply the operator to."""
    s, r = _sphere(lat), _radii(rad)
    kmax = math.pi * (1 << lat) / 1.2
    return torch.stack([_waves(s, r, rng, kmax) for _ in range(3)])


def _scalar(lat, rad, rng):
    return _waves(_sphere(lat), _radii(rad), rng, math.pi * (1 << lat) / 1.2)


def _profile(field, contrast):
    return torch.exp(0.5 * math.log(contrast) * field / field.abs().max())


def _coefficient(case, rng):
    """Viscosity: smooth with contrast 1e2 at the nodes, or per cell the same times lateral blocks of up to 1e4."""
    s, r = _sphere(case["lat"]), _radii(case["rad"])
    if not case["q0"]:
        return _profile(_waves(s, r, rng, 4.0), 100.0)
    c = _unit(s[:, :-1, :-1] + s[:, 1:, :-1] + s[:, :-1, 1:] + s[:, 1:, 1:])
    eta = _profile(_waves(c, 0.5 * (r[:-1] + r[1:]), rng, 4.0), 10.0)
    tiles = min(4, c.shape[1])
    edge = c.shape[1] // tiles
    f = np.where(rng.uniform(size=(10, tiles, tiles)) < 0.3, 10.0 ** rng.uniform(0.0, 4.0, (10, tiles, tiles)), 1.0)
    f = torch.tensor(f, device="cuda").repeat_interleave(edge, 1).repeat_interleave(edge, 2)
    return eta * f[..., None]


def _inputs(case, seed):
    """Every number a case is made of, as FP64 or FP32 device tensors."""
    rng = np.random.default_rng([seed, case["lat"], case["rad"]])
    lat, rad, op = case["lat"], case["rad"], case["op"]
    solver = op in ("precondition", "cg", "solve")
    dt = torch.float64 if solver else _dtype(case)
    x = {"k": _coefficient(case, rng).to(dt).contiguous()}
    if op == "galerkin":
        x["u"] = _velocity(lat - 1, rad - 1, rng)
    elif op == "gca_build":
        x["u1"], x["u2"] = _velocity(lat - 1, rad - 1, rng), _velocity(lat - 2, rad - 2, rng)
    else:
        x["u"] = _velocity(lat, rad, rng)
    if op == "vjp":
        x["lam"] = _velocity(lat, rad, rng)
    if op in ("stokes", "precondition"):
        x["p"] = _scalar(lat - 1, rad - 1, rng)
    if op == "solve":  # buoyancy of a smooth temperature with thermal noise
        s, r = _sphere(lat), _radii(rad)
        temp = _waves(s, r, rng, 6.0) + 0.01 * _waves(s, r, rng, math.pi * (1 << lat) / 1.2)
        x["u"] = temp[None] * torch.tensor(s, device="cuda").permute(3, 0, 1, 2)[..., None]
    for k in list(x):
        x[k] = x[k].to(dt).contiguous()
    return x


# ----------------------------------------------------------------------------------------------------------------
# State and pass
# ----------------------------------------------------------------------------------------------------------------
def _comps(v):
    return [v[c] for c in range(v.shape[0])]


def prepare(case, seed):
    x = _inputs(case, seed)
    op, lat, rad = case["op"], case["lat"], case["rad"]
    bcs = {"bc_cmb": case["cmb"], "bc_surface": case["surface"]}
    nlev = {"apply": 1, "vjp": 1, "stokes": 2, "galerkin": 2, "gca_build": 3}.get(op) or case["levels"]
    sh = T.Shell(lat, rad, num_levels=nlev, r_min=R_MIN, r_max=R_MAX)
    st = {"op": op, "shell": sh, "x": x}
    coef = {"k_cell" if case["q0"] else "k": x["k"]}
    if op in ("apply", "vjp"):
        st["A"] = T.EpsDivDiv(sh, -1, **coef, **bcs)
        st["out"] = torch.empty_like(x["u"])
        if op == "vjp":
            st["grad"] = torch.empty_like(x["k"])
    elif op == "stokes":
        st["A"] = T.Stokes(sh, -1, **coef, **bcs)
        st["in"] = _comps(x["u"]) + [x["p"]]
        st["out"] = [torch.empty_like(v) for v in st["in"]]
    elif op in ("galerkin", "gca_build"):
        st["A"] = T.EpsDivDiv(sh, -1, **coef, **bcs)
        st["coarse"] = []
        for l in range(2, nlev + 1):
            nl, nr = sh.dims(-l)
            shape = (10, nl - 1, nl - 1, nr - 1) if case["q0"] else (10, nl, nl, nr)
            one = torch.ones(shape, dtype=torch.float64, device="cuda")
            st["coarse"].append(T.EpsDivDiv(sh, -l, **{"k_cell" if case["q0"] else "k": one}, **bcs))
        if op == "galerkin":
            T.gca_build(st["A"], st["coarse"][0])
            st["out"] = torch.empty_like(x["u"])
            st["coarse"][0].apply(x["u"], st["out"])  # lays out the boundary-treated matrices once
        else:
            st["out"] = [torch.empty_like(x["u1"]), torch.empty_like(x["u2"])]
    elif op == "cg":
        st["solver"] = T.VelocitySolver(sh, eta=x["k"], **bcs, chebyshev_order=3, chebyshev_iterations=2,
                                        relative_tolerance=1e-8, absolute_tolerance=0.0,
                                        mixed_precision=int(case["dtype"] == "f32"))
        T.stokes_rhs_enforce(sh, -1, x["u"], **bcs)
        st["b"] = _comps(x["u"])
        st["out"] = [torch.zeros_like(v) for v in st["b"]]
    else:
        st["solver"] = T.StokesSolver(sh, eta=x["k"], **bcs, chebyshev_order=3, coarse_solver=T.COARSE_DENSE,
                                      relative_tolerance=1e-8, absolute_tolerance=0.0, max_iterations=3000,
                                      project_pressure_mean=1, mixed_precision=int(case["dtype"] == "f32"))
        if op == "precondition":
            st["b"] = _comps(x["u"]) + [x["p"]]
        else:
            f = torch.zeros_like(x["u"])
            T.vector_mass_apply(sh, -1, x["u"], f)
            T.stokes_rhs_enforce(sh, -1, f, **bcs)
            nl, nr = sh.dims(-2)
            st["b"] = _comps(f) + [torch.zeros((10, nl, nl, nr), dtype=torch.float64, device="cuda")]
        st["out"] = [torch.zeros_like(v) for v in st["b"]]
    return st


def run(st):
    op, x = st["op"], st["x"]
    if op == "apply":
        return st["A"].apply(x["u"], st["out"])
    if op == "stokes":
        return st["A"].apply(st["in"], st["out"])
    if op == "vjp":
        st["A"].vjp(x["u"], x["lam"], st["grad"], grad_u=st["out"])
        return [st["grad"], st["out"]]
    if op == "galerkin":
        return st["coarse"][0].apply(x["u"], st["out"])
    if op == "gca_build":
        c1, c2 = st["coarse"]
        T.gca_build(st["A"], c1)
        T.gca_build(c1, c2)
        return [c1.apply(x["u1"], st["out"][0]), c2.apply(x["u2"], st["out"][1])]
    if op == "precondition":
        return st["solver"].precondition(st["b"], st["out"])
    for v in st["out"]:
        v.zero_()
    st["solver"].solve(st["out"], st["b"])
    return st["out"]


# ----------------------------------------------------------------------------------------------------------------
# Work
# ----------------------------------------------------------------------------------------------------------------
_APPLY_FLOPS = 2 * 160  # per cell: two wedges of gradient, stress and its product with the six gradients


def _dims(case, down=0):
    nl, nr = (1 << (case["lat"] - down)) + 1, (1 << (case["rad"] - down)) + 1
    return 10 * nl * nl * nr, 10 * (nl - 1) ** 2 * (nr - 1)


def _stored_bytes(cells, item):
    return cells * 342 * item  # two symmetric 18 x 18 matrices


def _vcycle_work(case, item):
    """One V(2,2) cycle of order-3 Chebyshev smoothing from a zero guess: per level 11 smoother applies and one
    residual (5 of the smoother's on the way down), each with its vectors read and written once."""
    by = fl = 0.0
    for d in range(case["levels"] - 1):
        nodes, cells = _dims(case, d)
        vec = 3 * nodes * item
        applies = 12
        by += applies * 2 * vec + 12 * 5 * vec + 4 * vec  # operator, updates (b, invdiag, d, x in and out), transfers
        by += applies * (nodes * item if d == 0 else _stored_bytes(cells, item))
        fl += applies * (cells * _APPLY_FLOPS if d == 0 else cells * 342 * 4)
    return by, fl


def work(case):
    op, item = case["op"], 4 if case["dtype"] == "f32" else 8
    nodes, cells = _dims(case)
    pn = _dims(case, 1)[0]
    kn = cells if case["q0"] else nodes
    if op == "apply":
        return {"bytes": (6 * nodes + kn) * item, "flops": cells * _APPLY_FLOPS}
    if op == "stokes":
        return {"bytes": (6 * nodes + kn + 2 * pn) * item, "flops": cells * (_APPLY_FLOPS + 160)}
    if op == "vjp":
        return {"bytes": (9 * nodes + 2 * kn) * item, "flops": cells * (2 * _APPLY_FLOPS)}
    if op == "galerkin":
        cn, cc = _dims(case, 1)
        return {"bytes": _stored_bytes(cc, 8) + 6 * cn * 8, "flops": cc * 342 * 4}
    if op == "gca_build":
        (n1, c1), (n2, c2) = _dims(case, 1), _dims(case, 2)
        return {"bytes": kn * 8 + _stored_bytes(c1 + c2, 8) + 6 * (n1 + n2) * 8,
                "flops": cells * 2 * (171 * 8 + 300) + c1 * 2 * 2 * 2 * 18 * 18 * 6}
    # one preconditioner application / one Krylov iteration: V-cycle, B^T and the Schur step, then for an iteration
    # the operator in FP64 and the Gram-Schmidt of half a restart cycle of basis vectors (each read twice)
    vb, vf = _vcycle_work(case, item)
    pre = vb + (3 * nodes * 3 + 3 * pn) * 8
    if op == "precondition":
        return {"bytes": pre, "flops": vf + cells * 80}
    if op == "cg":
        its = 20
        return {"bytes": its * (vb + 13 * 3 * nodes * 8 + kn * 8), "flops": its * (vf + cells * _APPLY_FLOPS)}
    its = {3: 35, 4: 48, 5: 70, 6: 139}[case["lat"]]
    blk = (3 * nodes + pn) * 8
    return {"bytes": its * (pre + 2 * blk + kn * 8 + 2 * 16 * blk),
            "flops": its * (vf + cells * (_APPLY_FLOPS + 240) + 4 * 16 * blk / 8)}


# ----------------------------------------------------------------------------------------------------------------
# Tolerances: about four times the differences measured against `exact`, between repeated passes and between the
# FP64 and the mixed-precision form of the same call
# ----------------------------------------------------------------------------------------------------------------
def tolerance(case):
    op, f32 = case["op"], case["dtype"] == "f32"
    if op in ("apply", "stokes", "vjp"):
        if not f32:
            return {"rel": 4e-15, "max": 1e-13}
        # edge vectors of a wedge are differences of FP32 unit vectors and lose a bit per level
        h = 2.0 ** (case["lat"] - 6)
        return {"rel": max(1e-6, 1.7e-5 * h), "max": max(2e-5, 6.5e-4 * h)}
    if op in ("galerkin", "gca_build"):
        return {"rel": 4e-15, "max": 4e-14}
    if op == "precondition":
        return {"rel": 4e-7, "max": 5e-6} if f32 else {"rel": 2e-14}
    # a solution to 1e-8 moves with the iteration it stops at: 1.5e-8 (cg) and up to 2e-7 (solve) an iteration
    return {"rel": 6e-8} if op == "cg" else {"rel": 8e-7}


# ----------------------------------------------------------------------------------------------------------------
# The discretisation in 64 bits, wedge by wedge, from its definition
# ----------------------------------------------------------------------------------------------------------------
_WEDGE = [[(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (0, 1, 1)],
          [(1, 1, 0), (0, 1, 0), (1, 0, 0), (1, 1, 1), (0, 1, 1), (1, 0, 1)]]


def _corner(a, off, n):
    """Values of a (nx, ny, ...) lateral array at the given corner of every one of n x n cells."""
    return a[off[0]:off[0] + n, off[1]:off[1] + n]


def _node(a, off):
    """Values of a (..., nl, nl, nr) nodal array at one corner of every cell of a diamond."""
    nl, nr = a.shape[-3], a.shape[-1]
    return a[..., off[0]:off[0] + nl - 1, off[1]:off[1] + nl - 1, off[2]:off[2] + nr - 1]


class _Exact:
    """One level's wedges of one diamond at a time: gradients g (cells, 6, 3) and weights k |det J|."""

    def __init__(self, case):
        self.case = case
        self.sph = torch.tensor(_sphere(case["lat"]), device="cuda")
        self.r = torch.tensor(_radii(case["rad"]), device="cuda")

    def gradients(self, d, w):
        n = self.sph.shape[1] - 1
        p = [_corner(self.sph[d], o, n)[:, :, None] for o in _WEDGE[w][:3]]
        rm, h = 0.5 * (self.r[:-1] + self.r[1:])[:, None], 0.5 * (self.r[1:] - self.r[:-1])[:, None]
        j = torch.stack([(p[1] - p[0]) * rm, (p[2] - p[0]) * rm, (p[0] + p[1] + p[2]) / 3.0 * h], -1)
        ref = torch.tensor([[lx * 0.5, ly * 0.5, s * 0.5 / 3.0] for s in (-1.0, 1.0)
                            for lx, ly in ((-1.0, -1.0), (1.0, 0.0), (0.0, 1.0))], device="cuda", dtype=torch.float64)
        inv = torch.linalg.inv(j)
        return torch.einsum("nk,...ki->...ni", ref, inv), torch.linalg.det(j).abs()

    def weight(self, d, w, k):
        if self.case["q0"]:
            return k[d]
        return sum(_node(k[d], o) for o in _WEDGE[w]) / 6.0


def _stress(g, kw, u):
    """Nodal forces of the velocities u (..., 6, 3) on wedges with gradients g and weights kw."""
    grad = torch.einsum("...ni,...nj->...ij", g, u)
    sig = grad + grad.transpose(-1, -2)
    tr = torch.diagonal(grad, dim1=-2, dim2=-1).sum(-1)
    sig = (sig - (2.0 / 3.0) * tr[..., None, None] * torch.eye(3, device="cuda", dtype=torch.float64)) * kw[..., None, None]
    return torch.einsum("...ij,...nj->...ni", sig, g)


def _side_bc(case, rad):
    """Boundary condition of every node plane of a level with 2^rad layers."""
    b = [NEUMANN] * ((1 << rad) + 1)
    b[0], b[-1] = case["cmb"], case["surface"]
    return b


def _treat_input(u, sph, bc):
    v = u.clone()
    for r in (0, len(bc) - 1):
        if bc[r] == DIRICHLET:
            v[..., r] = 0.0
        elif bc[r] == FREESLIP:
            n = sph.permute(3, 0, 1, 2)
            v[..., r] = u[..., r] - (n * u[..., r]).sum(0) * n
    return v


def _treat_output(out, diag, u, sph, bc):
    """diag: (3, 10, nl, nl, nr) diagonal; on free-slip planes its first component is the normal stiffness."""
    for r in (0, len(bc) - 1):
        if bc[r] == DIRICHLET:
            out[..., r] = diag[..., r] * u[..., r]
        elif bc[r] == FREESLIP:
            n = sph.permute(3, 0, 1, 2)
            out[..., r] = out[..., r] + (diag[0, ..., r] * (n * u[..., r]).sum(0) - (n * out[..., r]).sum(0)) * n
    return out


def _diag_terms(g, kw, nrm):
    """Diagonal of the element matrices (..., 6, 3), and n^T A n in the direction nrm (..., 6, 3)."""
    gg = (g * g).sum(-1, keepdim=True)
    return kw[..., None, None] * (gg + g * g / 3.0), kw[..., None] * (gg[..., 0] + (nrm * g).sum(-1) ** 2 / 3.0)


def _scatter(out, d, w, f):
    """out[:, d] += f (cells..., 6, 3) at the wedge's nodes."""
    for i, o in enumerate(_WEDGE[w]):
        for c in range(3):
            _node(out[c, d], o).add_(f[..., i, c])


def _scatter_diag(diag, d, w, bc, dg, ann):
    for i, o in enumerate(_WEDGE[w]):
        for r in (0, len(bc) - 1):
            layer = r - o[2]
            if not 0 <= layer < len(bc) - 1:
                continue
            nl = diag.shape[2]
            for c in range(3):
                v = ann[..., layer, i] if bc[r] == FREESLIP else dg[..., layer, i, c]
                diag[c, d, o[0]:o[0] + nl - 1, o[1]:o[1] + nl - 1, r] += v


def _join(v, lat):
    """Sum over the copies of every node; v (ncomp, 10, nl, nl, nr)."""
    inv = _unique_columns(lat)
    f = v.reshape(v.shape[0], -1, v.shape[-1])
    s = torch.zeros((v.shape[0], int(inv.max()) + 1, v.shape[-1]), dtype=v.dtype, device=v.device)
    s.index_add_(1, inv, f)
    return s[:, inv].reshape(v.shape)


def _owned(lat):
    """One copy of every column (the first): (10, nl, nl) zeros and ones."""
    inv = _unique_columns(lat).cpu().numpy()
    first = np.zeros(inv.size)
    first[np.unique(inv, return_index=True)[1]] = 1.0
    nl = (1 << lat) + 1
    return torch.tensor(first.reshape(10, nl, nl), device="cuda")


def _rotation_penalty(u, sph, r, lat):
    """With free slip on both sides: 1e-7 sum_i (n_i^T u) n_i over the orthonormalised rigid rotations, added on
    every copy before the copies are summed."""
    x = sph[..., None, :] * r[:, None]
    modes = []
    for i in range(3):
        m = torch.zeros_like(u)
        a, b = (i + 1) % 3, (i + 2) % 3
        m[a], m[b] = -x[..., b], x[..., a]
        modes.append(m)
    own = _owned(lat)[None, ..., None]
    dot = lambda a, b: (a * b * own).sum()  # noqa: E731
    basis = []
    for m in modes:
        for q in basis:
            m = m - dot(m, q) * q
        basis.append(m / torch.sqrt(dot(m, m)))
    return 1e-7 * sum(dot(q, u) * q for q in basis)


def _apply_exact(case, k, u, joined=True):
    E = _Exact(case)
    bc = _side_bc(case, case["rad"])
    v, out, diag = _treat_input(u, E.sph, bc), torch.zeros_like(u), torch.zeros_like(u)
    n = E.sph.shape[1] - 1
    for d in range(10):
        for w in range(2):
            g, det = E.gradients(d, w)
            kw = det * E.weight(d, w, k)
            uw = torch.stack([_node(v[:, d], o) for o in _WEDGE[w]], -1).permute(1, 2, 3, 4, 0)
            _scatter(out, d, w, _stress(g, kw, uw))
            nrm = torch.stack([_corner(E.sph[d], o, n) for o in _WEDGE[w]], -2)[:, :, None]
            _scatter_diag(diag, d, w, bc, *_diag_terms(g, kw, nrm))
    _treat_output(out, diag, u, E.sph, bc)
    if case["cmb"] == FREESLIP and case["surface"] == FREESLIP:
        out = out + _rotation_penalty(u, E.sph, E.r, case["lat"])
    return _join(out, case["lat"]) if joined else out


def _vjp_exact(case, k, u, lam):
    E = _Exact(case)
    bc = _side_bc(case, case["rad"])
    vu, vl = _treat_input(u, E.sph, bc), _treat_input(lam, E.sph, bc)
    grad = torch.zeros_like(k)
    n = E.sph.shape[1] - 1
    for d in range(10):
        for w in range(2):
            g, det = E.gradients(d, w)
            kw = det * k[d]
            at = lambda a: torch.stack([_node(a[:, d], o) for o in _WEDGE[w]], -1).permute(1, 2, 3, 4, 0)  # noqa: E731
            val = (_stress(g, kw, at(vu)) * at(vl)).sum((-1, -2))
            nrm = torch.stack([_corner(E.sph[d], o, n) for o in _WEDGE[w]], -2)[:, :, None].expand(g.shape)
            dg, ann = _diag_terms(g, kw, nrm)
            ru, rl = at(u), at(lam)
            for layer, first, kind in ((0, 0, bc[0]), (-1, 3, bc[-1])):
                s = slice(first, first + 3)
                a, b = ru[:, :, layer, s], rl[:, :, layer, s]
                if kind == DIRICHLET:
                    val[:, :, layer] += (dg[:, :, layer, s] * a * b).sum((-1, -2))
                elif kind == FREESLIP:
                    m = nrm[:, :, layer, s]
                    val[:, :, layer] += (ann[:, :, layer, s] * (m * a).sum(-1) * (m * b).sum(-1)).sum(-1)
            grad[d] += val
    return grad


def _pressure_weights(case):
    """Per fine wedge (lateral parity x, y, wedge w) and radial parity: weights of the six coarse pressure nodes at
    the fine wedge's centroid. The coarse node of wedge node i is (x / 2, y / 2, r / 2) + its offset."""
    lat = {0: (2 / 3, 1 / 6, 1 / 6), 1: (1 / 6, 2 / 3, 1 / 6), 2: (1 / 6, 1 / 6, 2 / 3), 3: (1 / 3, 1 / 3, 1 / 3)}
    which = [[[0, 1], [2, 3]], [[3, 2], [1, 0]]]  # [w][y parity][x parity]
    return lambda w, py, px, pr: [a * b for b in ((0.75, 0.25) if pr == 0 else (0.25, 0.75))
                                  for a in lat[which[w][py][px]]]


def _coupling_exact(case, u, p):
    """(B^T p before the copies are summed, B u)."""
    E = _Exact(case)
    bc = _side_bc(case, case["rad"])
    wts = _pressure_weights(case)
    v = _treat_input(u, E.sph, bc)
    bt, b = torch.zeros_like(u), torch.zeros_like(p)
    nc, rc = p.shape[1] - 1, p.shape[-1] - 1
    for d in range(10):
        for w in range(2):
            g, det = E.gradients(d, w)
            uw = torch.stack([_node(v[:, d], o) for o in _WEDGE[w]], -1).permute(1, 2, 3, 4, 0)
            div = -det * (g * uw).sum((-1, -2))
            pi = torch.zeros_like(det)
            for px in (0, 1):
                for py in (0, 1):
                    for pr in (0, 1):
                        for i, o in enumerate(_WEDGE[w]):
                            wt = wts(w, py, px, pr)[i]
                            pi[px::2, py::2, pr::2] += wt * p[d, o[0]:o[0] + nc, o[1]:o[1] + nc, o[2]:o[2] + rc]
                            b[d, o[0]:o[0] + nc, o[1]:o[1] + nc, o[2]:o[2] + rc] += wt * div[px::2, py::2, pr::2]
            _scatter(bt, d, w, (-det * pi)[..., None, None] * g)
    bt = _treat_input(bt, E.sph, bc)  # Dirichlet rows zero, free-slip rows tangential
    return bt, _join(b[None], case["lat"] - 1)[0]


def _interpolation(h, w, outer):
    """6 x 6 interpolation from the coarse wedge's nodes to the nodes of fine wedge w of fine hex h = (hx, hy, hr).
    A node in the top plane of the coarse hex between two node columns takes the coarse wedge's bottom values, except
    on the outermost shell."""
    P = np.zeros((6, 6))
    for i, o in enumerate(_WEDGE[w]):
        x, y, r = h[0] + o[0], h[1] + o[1], h[2] + o[2]
        if x % 2 == 0 and y % 2 == 0:
            if r % 2 == 0:
                P[i, i] = 1.0
            else:
                P[i, i % 3] = P[i, i % 3 + 3] = 0.5
            continue
        pair = (0, 2) if x % 2 == 0 else ((0, 1) if y % 2 == 0 else (1, 2))
        for c in pair:
            if r % 2 == 1:
                P[i, c] = P[i, c + 3] = 0.25
            else:
                P[i, c + (3 if r == 2 and outer else 0)] = 0.5
    return torch.tensor(P, device="cuda")


def _coarsen(parts):
    """Galerkin coarsening of one diamond: parts[w] is a list of (gradients, weights) on the fine cells; the coarse
    wedge t holds P^T g of the fine wedges in it."""
    out = [[], []]
    for hx in (0, 1):
        for hy in (0, 1):
            for hr in (0, 1):
                for w in (0, 1):
                    t = (1 if hx and hy else 0) if w == 0 else (0 if not hx and not hy else 1)
                    for g, kw in parts[w]:
                        gg, kk = g[hx::2, hy::2, hr::2], kw[hx::2, hy::2, hr::2]
                        h = torch.einsum("nc,...nj->...cj", _interpolation((hx, hy, hr), w, False), gg)
                        if hr == 1:
                            h[:, :, -1] = torch.einsum("nc,...nj->...cj", _interpolation((hx, hy, hr), w, True),
                                                       gg[:, :, -1])
                        out[t].append((h, kk.contiguous()))
    return out


def _galerkin_exact(case, k, us):
    """Applies of the Galerkin operators one, two, ... levels down, to us[0], us[1], ..."""
    E = _Exact(case)
    res = []
    acc = [(torch.zeros_like(u), torch.zeros_like(u)) for u in us]
    for d in range(10):
        parts = []
        for w in range(2):
            g, det = E.gradients(d, w)
            parts.append([(g, det * E.weight(d, w, k))])
        for i, u in enumerate(us):
            parts = _coarsen(parts)
            s = 1 << (i + 1)
            sph = E.sph[:, ::s, ::s]
            bc = _side_bc(case, case["rad"] - i - 1)
            v = _treat_input(u[:, d:d + 1], sph[d:d + 1], bc)[:, 0]
            n = sph.shape[1] - 1
            out, diag = acc[i]
            for w in range(2):
                uw = torch.stack([_node(v, o) for o in _WEDGE[w]], -1).permute(1, 2, 3, 4, 0)
                nrm = torch.stack([_corner(sph[d], o, n) for o in _WEDGE[w]], -2)[:, :, None]
                for g, kw in parts[w]:
                    _scatter(out, d, w, _stress(g, kw, uw))
                    _scatter_diag(diag, d, w, bc, *_diag_terms(g, kw, nrm))
    for i, u in enumerate(us):
        s = 1 << (i + 1)
        sph, lat, rad = E.sph[:, ::s, ::s], case["lat"] - i - 1, case["rad"] - i - 1
        out = _treat_output(acc[i][0], acc[i][1], u, sph, _side_bc(case, rad))
        if case["cmb"] == FREESLIP and case["surface"] == FREESLIP:
            out = out + _rotation_penalty(u, sph, E.r[::s], lat)
        res.append(_join(out, lat))
    return res


def exact(case, seed):
    """Results of the operators in 64 bits. The solvers and the preconditioner have none: they are iterations whose
    result is defined by their steps, not by a closed expression."""
    op = case["op"]
    if op in ("precondition", "cg", "solve"):
        return None
    x = {k: v.double() for k, v in _inputs(case, seed).items()}
    if op == "apply":
        return _apply_exact(case, x["k"], x["u"])
    if op == "vjp":
        return [_vjp_exact(case, x["k"], x["u"], x["lam"]), _apply_exact(case, x["k"], x["lam"])]
    if op == "stokes":
        bt, b = _coupling_exact(case, x["u"], x["p"])
        # the operator's free-slip penalty is part of A, which is added to B^T p before the copies are summed
        f = _join(_apply_exact(case, x["k"], x["u"], joined=False) + bt, case["lat"])
        return [f[0], f[1], f[2], b]
    if op == "galerkin":
        return _galerkin_exact(case, x["k"], [x["u"]])[0]
    return _galerkin_exact(case, x["k"], [x["u1"], x["u2"]])
