"""Performance cases of the SolverV4 state solve and design update.

Each case is one call (or one short chain of calls) that a program using this
package makes, through its public entry points:

* ``matvec``    y = K(E) u, ``TopoContext.matvec`` (FP64, FP32 and BF16 input);
* ``smooth``    one fused Chebyshev step of the mixed-precision smoother,
                ``TopoContext.level0_apply(..., "cheb")``;
* ``vcycle``    one multigrid V-cycle on a hierarchy the program keeps,
                ``TopoContext.gmg_apply``;
* ``precond``   hierarchy set-up for new moduli, then one V-cycle (what a design
                loop pays before its first Krylov step);
* ``state``     a whole FP64 state solve (moduli, set-up, PCG, compliance,
                sensitivity), ``StateSolver.solve``;
* ``block``     one density, several load cases, ``StateSolver.solve_block``;
* ``gradient``  filtered compliance and its gradient with respect to FP32
                design variables through autograd (forward and backward);
* ``design``    the filtered design update: H^T of the sensitivities, OC with
                the filtered volume, H of the new design;
* ``projected`` the same with the Heaviside projection.

Meshes run from 24x12x6 (the smallest configuration) to 160x80x80 (1,024,000
elements), uneven extents among them.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from topogpu_b200.autograd import compliance, density_filter
from topogpu_b200.bc import cantilever_edge_load, face_point_loads
from topogpu_b200.context import TopoContext
from topogpu_b200.state import StateSolver

DEV = "cuda"
EMIN = 1e-9
CHEB = {"s": 1.0, "c1": 0.29, "c2": 0.87, "ax": 1.0}  # a step of the degree-3 smoother, D^-1 scaled by lambda_max ~ 1
MOVE, RHO_MIN, VOLFRAC = 0.2, 1e-3, 0.30


def listed():
    return [
        # the smallest call: a Krylov method of the user's own on the smallest configuration
        {"name": "matvec f64 24x12x6", "kind": "matvec", "dtype": "f64", "nx": 24, "ny": 12, "nz": 6},
        # the operator benchmark's mesh
        {"name": "matvec f32 192x96x48", "kind": "matvec", "dtype": "f32", "nx": 192, "ny": 96, "nz": 48},
        # the smoother of the mixed-precision hierarchy at one million elements
        {"name": "smooth bf16 160x80x80", "kind": "smooth", "nx": 160, "ny": 80, "nz": 80},
        # one preconditioner application on an uneven mesh
        {"name": "vcycle fp32 61x30x23", "kind": "vcycle", "precision": "fp32", "nx": 61, "ny": 30, "nz": 23},
        # a design loop's new hierarchy and first preconditioned residual at one million elements
        {"name": "precond mixed 160x80x80", "kind": "precond", "precision": "mixed", "nx": 160, "ny": 80, "nz": 80},
        # whole FP64 state solves: the smallest configuration and the differentiation configuration
        {"name": "state fp64 24x12x6", "kind": "state", "nx": 24, "ny": 12, "nz": 6},
        {"name": "state fp64 48x24x24", "kind": "state", "nx": 48, "ny": 24, "nz": 24},
        # eight load cases on one density
        {"name": "block fp64 96x48x48", "kind": "block", "loads": 8, "nx": 96, "ny": 48, "nz": 48},
        # gradient-based design with FP32 variables: one million elements, and one of many small meshes
        {"name": "gradient mixed 160x80x80", "kind": "gradient", "precision": "mixed", "rmin": 2.0,
         "nx": 160, "ny": 80, "nz": 80},
        {"name": "gradient mixed 43x21x17", "kind": "gradient", "precision": "mixed", "rmin": 1.5,
         "nx": 43, "ny": 21, "nz": 17},
        # design updates
        {"name": "design 160x80x80", "kind": "design", "rmin": 2.0, "nx": 160, "ny": 80, "nz": 80},
        {"name": "projected 96x48x48", "kind": "projected", "rmin": 2.0, "beta": 8.0, "nx": 96, "ny": 48, "nz": 48},
    ]


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "smooth", "vcycle", "precond", "state", "block", "gradient", "design",
                       "projected"])
    top = {"block": 96, "state": 64, "projected": 112}.get(kind, 160)
    nx = int(round(math.exp(rng.uniform(math.log(16), math.log(top)))))
    ny = max(8, int(round(nx * rng.uniform(0.4, 0.5))))
    nz = max(6 if kind in ("matvec", "smooth", "design", "projected") else 8, int(round(nx * rng.uniform(0.2, 0.5))))
    case = {"kind": kind, "nx": nx, "ny": ny, "nz": nz}
    if kind == "matvec":
        case["dtype"] = rng.choice(["f64", "f32", "bf16"])
    elif kind in ("vcycle", "precond", "gradient"):
        case["precision"] = rng.choice(["mixed", "mixed", "fp32"])
    elif kind == "block":
        case["loads"] = rng.randint(2, 8)
    if kind in ("gradient", "design", "projected"):
        case["rmin"] = rng.choice([1.5, 2.0, 2.3, 3.0])
    if kind == "projected":
        case["beta"] = rng.choice([1.0, 4.0, 8.0])
    return case


# ------------------------------------------------------------------ inputs
def _nel(case):
    return case["nx"], case["ny"], case["nz"]


def _levels(nel):
    """Levels of a factor-2 hierarchy whose coarsest grid keeps a few elements per direction."""
    k, m = 1, min(nel)
    while m >= 4 and k < 4:
        m //= 2
        k += 1
    return k


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rand(n, g, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(n, generator=g, dtype=torch.float64, device=DEV)


def _randn(n, g):
    return torch.randn(n, generator=g, dtype=torch.float64, device=DEV)


def _density(nel, seed):
    """An intermediate design: a smooth random field of a few waves around the
    volume fraction, with grey transitions, bounded away from void."""
    g = _gen(seed)
    ax = [torch.linspace(0.0, 1.0, n, dtype=torch.float64, device=DEV) for n in nel]
    X, Y, Z = torch.meshgrid(*ax, indexing="ij")
    f = torch.zeros(nel, dtype=torch.float64, device=DEV)
    for _ in range(6):
        w = _rand(7, g)
        f += (0.4 + 0.6 * w[6]) * torch.sin(2 * math.pi * ((1 + 3 * w[0]) * X + (1 + 2 * w[1]) * Y
                                                            + (1 + 2 * w[2]) * Z + w[3]))
    f = f / f.abs().max()
    noise = _rand(f.numel(), g, -0.02, 0.02).view(nel)
    return (VOLFRAC + 0.35 * f + noise).clamp(0.08, 1.0).reshape(-1).contiguous()


def _moduli(rho):
    return EMIN + (1.0 - EMIN) * rho ** 3


def _solver(case, seed, precision, tol):
    nel = _nel(case)
    mask, F = cantilever_edge_load(nel)
    return StateSolver(nel, mask, F, n_levels=_levels(nel), precision=precision, fine_degree=3, coarse_degree=2,
                       tol=tol, maxiter=800, warm_start=False)


def _sensitivities(rho, seed):
    """Compliance sensitivities as a state solve gives them: element energies over several decades."""
    g = _gen(seed + 1)
    return -3.0 * rho ** 2 * torch.exp(1.5 * _randn(rho.numel(), g))


def _vectors(nel, seed):
    """The cantilever's mask, moduli of an iid density (the operator benchmark's) and a normal vector."""
    mask, F = cantilever_edge_load(nel)
    g = _gen(seed)
    E = _moduli(_rand(int(np.prod(nel)), g, 1e-3, 1.0))
    m = torch.as_tensor(mask, device=DEV)
    return m, torch.as_tensor(F, device=DEV), E, _randn(m.numel(), g) * m, g


def prepare(case, seed):
    kind, nel = case["kind"], _nel(case)
    st = {"kind": kind, "case": case}
    if kind in ("matvec", "smooth"):
        m, F, E, u, g = _vectors(nel, seed)
        st["ctx"] = TopoContext(nel, n_levels=1, mode="mixed" if kind == "smooth" else "fp64")
        st["ctx"].set_problem(m, F)
        dt = {"f64": torch.float64, "f32": torch.float32, "bf16": torch.bfloat16}[case.get("dtype", "f32")]
        st["u"] = u.to(dt)
        st["E"] = E if dt == torch.float64 else E.float()
        if kind == "smooth":
            n = u.numel()
            st["r"], st["x"] = (_randn(n, g) * m).float(), (_randn(n, g) * m).float()
            st["dinv"] = (_rand(n, g, 0.2, 1.0) * m).float()
            st["d"] = torch.empty_like(st["r"])
    elif kind in ("vcycle", "precond"):
        st["solver"] = _solver(case, seed, case["precision"], 1e-5)
        st["E"] = _moduli(_density(nel, seed))
        r = _randn(st["solver"].ctx.ndof, _gen(seed + 1)) * st["solver"].free_mask
        st["r"] = r.to(st["solver"].ctx.vec_dtype)
        if kind == "vcycle":
            st["solver"].ctx.gmg_setup(st["E"])
    elif kind == "state":
        st["solver"] = _solver(case, seed, "fp64", 1e-8)
        st["rho"] = _density(nel, seed)
    elif kind == "block":
        st["solver"] = _solver(case, seed, "fp64", 1e-5)
        st["rho"] = _density(nel, seed)
        st["loads"] = torch.as_tensor(face_point_loads(nel, case["loads"], seed), device=DEV)
    elif kind == "gradient":
        st["solver"] = _solver(case, seed, case["precision"], 1e-5)
        st["x"] = _density(nel, seed).float().requires_grad_(True)
    elif kind in ("design", "projected"):
        st["ctx"] = TopoContext(nel, n_levels=1, mode="fp64")
        st["rho"] = _density(nel, seed)
        st["dc"] = _sensitivities(st["rho"], seed)
        if kind == "design":
            st["colsum"] = st["ctx"].filter(case["rmin"], torch.ones_like(st["rho"]), transpose=True)
    return st


def run(st):
    kind, case = st["kind"], st["case"]
    if kind == "matvec":
        return st["ctx"].matvec(st["u"], st["E"])
    if kind == "smooth":
        st["ctx"].level0_apply(st["u"], st["E"], "cheb", r=st["r"], x=st["x"], d_out=st["d"], dinv=st["dinv"],
                               u_fp32_to_bf16=True, **CHEB)
        return {"r": st["r"], "x": st["x"], "d": st["d"]}
    if kind == "vcycle":
        return st["solver"].ctx.gmg_apply(st["r"])
    if kind == "precond":
        st["solver"].ctx.gmg_setup(st["E"])
        return st["solver"].ctx.gmg_apply(st["r"])
    if kind == "state":
        c, dc = st["solver"].solve(st["rho"], 3.0)
        return {"compliance": c, "dc": dc, "u": st["solver"].displacement()}
    if kind == "block":
        c, U = st["solver"].solve_block(st["rho"], st["loads"], 3.0)
        return {"compliance": c, "U": U}
    if kind == "gradient":
        x, sol = st["x"], st["solver"]
        x.grad = None
        c = compliance(density_filter(x.double(), sol.ctx, case["rmin"]), sol)
        c.backward()
        return {"compliance": float(c.detach()), "grad": x.grad}
    ctx, rmin, rho = st["ctx"], case["rmin"], st["rho"]
    if kind == "design":
        dcd = ctx.filter(rmin, st["dc"], transpose=True)
        new, _ = ctx.oc_filtered(rho, dcd, st["colsum"], st["colsum"], VOLFRAC, MOVE, RHO_MIN)
        return {"dc": dcd, "rho": new, "rho_phys": ctx.filter(rmin, new)}
    phys, dh = ctx.heaviside(ctx.filter(rmin, rho), case["beta"], 0.5)
    dcd = ctx.filter(rmin, st["dc"] * dh, transpose=True)
    dvd = ctx.filter(rmin, dh, transpose=True)
    new, _ = ctx.oc_projected(rmin, rho, dcd, dvd, case["beta"], 0.5, VOLFRAC, MOVE, RHO_MIN)
    return {"phys": phys, "dc": dcd, "dv": dvd, "rho": new}


# -------------------------------------------------------------------- work
def _ku(nel, vec_bytes, e_bytes):
    """Bytes and operations of one K u: vectors as given per DoF, moduli and
    the one-byte mask once; per element 24 adds in each of three directions
    for the sums and differences of corner values and for their transpose,
    eight 3x3 products and the scaling."""
    nodes, elems = (nel[0] + 1) * (nel[1] + 1) * (nel[2] + 1), nel[0] * nel[1] * nel[2]
    return np.array([3.0 * nodes * (vec_bytes + 1) + elems * e_bytes, 312.0 * elems])


def _coarse(nel, vec_bytes, c_bytes):
    """One 27-point block stencil product: 243 coefficients per node and the vectors."""
    nodes = (nel[0] + 1) * (nel[1] + 1) * (nel[2] + 1)
    return np.array([nodes * (243.0 * c_bytes + 3.0 * vec_bytes), 486.0 * nodes])


def _halve(nel):
    return tuple(max(1, n // 2) for n in nel)


def _vcycle(nel, levels, s, c):
    """Degree-3 (fine) and degree-2 (coarse) smoothing before and after, one
    residual and one update by the coarse correction per level; s: bytes of a
    vector entry, c: bytes of a coarse coefficient."""
    w = 4 * _ku(nel, 7 * s, s) + 2 * _ku(nel, 3 * s, s)
    for _ in range(1, levels - 1):
        nel = _halve(nel)
        w = w + 2 * _coarse(nel, 7 * s, c) + 2 * _coarse(nel, 3 * s, c)
    nel = _halve(nel)
    n, band = 3.0 * (nel[0] + 1) * (nel[1] + 1) * (nel[2] + 1), 3.0 * (nel[1] + 2) * (nel[2] + 2)
    return w + np.array([2 * n * band * s, 4 * n * band])


def _setup(nel, levels):
    """Moduli read, coarse FP64 operators written and read once, band factorisation of the coarsest level."""
    e = nel[0] * nel[1] * nel[2]
    w = np.array([8.0 * e, 0.0])
    for _ in range(1, levels):
        nel = _halve(nel)
        nodes = (nel[0] + 1) * (nel[1] + 1) * (nel[2] + 1)
        w = w + np.array([2 * 243 * 8.0 * nodes, 8 * 486.0 * nodes])
    band = 3.0 * (nel[1] + 2) * (nel[2] + 2)
    return w + np.array([0.0, 3.0 * (nel[0] + 1) * (nel[1] + 1) * (nel[2] + 1) * band * band])


def work(case):
    kind, nel = case["kind"], _nel(case)
    levels, e = _levels(nel), nel[0] * nel[1] * nel[2]
    if kind == "matvec":
        s = {"f64": (16, 8), "f32": (8, 4), "bf16": (6, 4)}[case["dtype"]]
        w = _ku(nel, *s)
    elif kind == "smooth":
        w = _ku(nel, 28, 4)
    elif kind in ("vcycle", "precond"):
        w = _vcycle(nel, levels, 4, 2 if case["precision"] == "mixed" else 4)
        w = w + (_setup(nel, levels) if kind == "precond" else 0.0)
    elif kind in ("state", "gradient"):
        # a dozen preconditioned iterations (more at tighter tolerance), sensitivity and filter
        s = 8 if kind == "state" else 4
        c = 2 if case.get("precision") == "mixed" else s
        its = 20 if kind == "state" else 12
        w = _setup(nel, levels) + its * (_vcycle(nel, levels, s, c) + _ku(nel, 6 * s, s)) + _ku(nel, 8, 24)
    elif kind == "block":
        w = _setup(nel, levels) + 10 * case["loads"] * (_vcycle(nel, levels, 8, 8) + _ku(nel, 64, 8 / case["loads"]))
    else:
        # the fields in and out of each filter, and one pass of the volume bracket
        taps = 4.0 / 3.0 * math.pi * case["rmin"] ** 3
        n = 3 if kind == "design" else 6
        w = np.array([(16.0 * n + 40.0) * e, (2 * taps * n + 60.0) * e])
    return {"bytes": float(w[0]), "flops": float(w[1])}


# ------------------------------------------------------- values in 64 bits
_CORNERS = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0], [0, 1, 0], [0, 0, 1], [1, 0, 1], [1, 1, 1], [0, 1, 1]])


def _hex_stiffness(nu=0.3):
    """24x24 stiffness of the trilinear cube of edge 2 (E = 1) by 2x2x2 Gauss quadrature."""
    lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 0.5 / (1 + nu)
    D = np.zeros((6, 6))
    D[:3, :3] = lam
    D[np.arange(3), np.arange(3)] += 2 * mu
    D[np.arange(3, 6), np.arange(3, 6)] = mu
    sg = 2.0 * _CORNERS - 1.0
    K = np.zeros((24, 24))
    for p in sg / math.sqrt(3.0):
        one = 1.0 + sg * p
        dN = np.stack([sg[:, k] * one[:, (k + 1) % 3] * one[:, (k + 2) % 3] / 8.0 for k in range(3)], axis=1)
        B = np.zeros((6, 24))
        for a in range(8):
            dx, dy, dz = dN[a]
            B[:, 3 * a:3 * a + 3] = [[dx, 0, 0], [0, dy, 0], [0, 0, dz], [dy, dx, 0], [0, dz, dy], [dz, 0, dx]]
        K += B.T @ D @ B
    return torch.as_tensor(K, device=DEV)


def _edof(nel):
    nx, ny, nz = nel
    ex, ey, ez = torch.meshgrid(*(torch.arange(n, device=DEV) for n in nel), indexing="ij")
    c = torch.as_tensor(_CORNERS, device=DEV)
    node = ((ex.reshape(-1, 1) + c[:, 0]) * (ny + 1) + ey.reshape(-1, 1) + c[:, 1]) * (nz + 1) + ez.reshape(-1, 1) + c[:, 2]
    return (3 * node.unsqueeze(2) + torch.arange(3, device=DEV)).reshape(-1, 24)


def _free(nel):
    m = torch.ones(3 * (nel[0] + 1) * (nel[1] + 1) * (nel[2] + 1), dtype=torch.float64, device=DEV)
    m[:3 * (nel[1] + 1) * (nel[2] + 1)] = 0.0
    return m


def _apply(edof, KE, E, m, u):
    y = torch.zeros_like(u)
    for a in range(0, edof.shape[0], 262144):
        ed = edof[a:a + 262144]
        y.index_add_(0, ed.reshape(-1), ((u[ed] @ KE) * E[a:a + 262144, None]).reshape(-1))
    return y * m


def _solve64(nel, E, F):
    """Diagonally preconditioned conjugate gradients in 64 bits to a residual of 1e-13."""
    KE, edof, m = _hex_stiffness(), _edof(nel), _free(nel)
    d = torch.zeros_like(m).index_add_(0, edof.reshape(-1), (torch.diagonal(KE)[None, :] * E[:, None]).reshape(-1))
    b = F * m
    x, r = torch.zeros_like(b), b.clone()
    z = r / d
    p, rz = z.clone(), torch.dot(r, z)
    for it in range(20000):
        q = _apply(edof, KE, E, m, p)
        a = rz / torch.dot(p, q)
        x, r = x + a * p, r - a * q
        z = r / d * m
        new = torch.dot(r, z)
        p, rz = z + (new / rz) * p, new
        if it % 50 == 49 and float(r.norm()) <= 1e-13 * float(b.norm()):
            break
    ce = ((x[edof] @ KE) * x[edof]).sum(dim=1)
    return x, ce


def _hat(nel, rmin):
    """The linear-hat filter as functions H x and H^T x: weights rmin - distance of the element centres, rows normalised."""
    R = int(math.floor(rmin))
    taps = [(i, j, k, rmin - math.sqrt(i * i + j * j + k * k)) for i in range(-R, R + 1) for j in range(-R, R + 1)
            for k in range(-R, R + 1) if i * i + j * j + k * k == 0 or math.sqrt(i * i + j * j + k * k) <= rmin - 1e-10]
    pad = torch.zeros([n + 2 * R for n in nel], dtype=torch.float64, device=DEV)

    def conv(x):
        p = pad.clone()
        p[R:R + nel[0], R:R + nel[1], R:R + nel[2]] = x.view(nel)
        y = torch.zeros(nel, dtype=torch.float64, device=DEV)
        for i, j, k, w in taps:
            y += w * p[R + i:R + i + nel[0], R + j:R + j + nel[1], R + k:R + k + nel[2]]
        return y.reshape(-1)

    rows = conv(torch.ones(int(np.prod(nel)), dtype=torch.float64, device=DEV))
    return (lambda x: conv(x) / rows), (lambda x: conv(x / rows))


def _bisect(rho, dc, dv, volume):
    """run_simp's bisection on the multiplier; the design of the last one evaluated."""
    lo, hi, k, new = 0.0, 1e9, 0, rho
    while hi - lo >= 1e-9 and k < 100:
        lm = 0.5 * (lo + hi)
        new = rho * torch.sqrt(dc.clamp(max=-1e-12).neg() / (lm * dv.clamp(min=1e-12)))
        new = torch.minimum(torch.maximum(new, rho - MOVE), rho + MOVE).clamp(RHO_MIN, 1.0)
        lo, hi = (lm, hi) if float(volume(new)) > VOLFRAC else (lo, lm)
        k += 1
    return new


def exact(case, seed):
    kind, nel = case["kind"], _nel(case)
    if kind in ("matvec", "smooth"):
        m, _, E, u, g = _vectors(nel, seed)
        m = m.double()
        KE = _hex_stiffness()
        if kind == "smooth" or case["dtype"] != "f64":
            E = E.float().double()
        if kind == "smooth" or case["dtype"] == "bf16":
            # the BF16 operator is defined on BF16-rounded u and KE
            KE, full, u = KE.float().bfloat16().double(), u.float().double(), u.float().bfloat16().double()
        elif case["dtype"] == "f32":
            u = u.float().double()
        y = _apply(_edof(nel), KE, E, m, u)
        if kind == "matvec":
            return y
        n = u.numel()
        r, x = (_randn(n, g) * m).float().double(), (_randn(n, g) * m).float().double()
        dinv = (_rand(n, g, 0.2, 1.0) * m).float().double()
        r = r - CHEB["s"] * y
        d = CHEB["c1"] * full + CHEB["c2"] * dinv * r
        return {"r": r, "x": x + CHEB["ax"] * d, "d": d}
    if kind == "state":
        rho = _density(nel, seed)
        F = torch.as_tensor(cantilever_edge_load(nel)[1], device=DEV)
        u, ce = _solve64(nel, _moduli(rho), F)
        return {"compliance": float(torch.dot(F, u)), "dc": -3.0 * (1.0 - EMIN) * rho ** 2 * ce, "u": u}
    if kind in ("design", "projected"):
        rho = _density(nel, seed)
        dc = _sensitivities(rho, seed)
        H, Ht = _hat(nel, case["rmin"])
        if kind == "design":
            dcd, col = Ht(dc), Ht(torch.ones_like(rho))
            new = _bisect(rho, dcd, col, lambda v: torch.dot(v, col) / v.numel())
            return {"dc": dcd, "rho": new, "rho_phys": H(new)}
        b = case["beta"]
        den = math.tanh(0.5 * b) + math.tanh(0.5 * b)
        t = torch.tanh(b * (H(rho) - 0.5))
        dh = b * (1.0 - t * t) / den
        dcd, dvd = Ht(dc * dh), Ht(dh)
        new = _bisect(rho, dcd, dvd, lambda v: ((math.tanh(0.5 * b) + torch.tanh(b * (H(v) - 0.5))) / den).mean())
        return {"phys": (math.tanh(0.5 * b) + t) / den, "dc": dcd, "dv": dvd, "rho": new}
    # a V-cycle is an approximate inverse of its own making, and a solve that
    # stops at 1e-5 has that tolerance in every digit after: no value of 64 bits
    return None
