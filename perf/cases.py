"""Performance cases: calls of the residual library as programs make them.

Each case is one pass through the public Python API on device tensors, with
the library on torch's stream: a state goes in, a residual, an advanced state
or an adjoint comes out.  ``listed`` names the cases, ``draw`` gives further
ones of the same ranges, ``prepare`` the inputs and the solver that a program
keeps, ``run`` one pass, ``work`` the bytes and operations a pass cannot do
without, ``exact`` the same outputs in plain 64-bit torch.

A case is a dict of
  op         residual | step | vjp | step_vjp | batch
  etype      quad | cyl | hex | tri       (cyl: O-mesh of nine-node quads)
  nx, ny, nz cells (cyl: radial, circumferential); tri has nx * nx * 2 elements
  P          polynomial order
  viscous, flux (rusanov | roe), beta (LDG), precision (fp64 | mixed)
  jitter     interior nodes moved by this share of the cell size
  steps      time steps of op "step" and "batch"
  cases      (batch) number of meshes; nx then is the largest mesh's size
"""
from __future__ import annotations

import collections
import functools
import math

import numpy as np
import torch

from zefr_b200 import meshgen
from zefr_b200.batch import Batch
from zefr_b200.solver import FRSolver, make_params

GAMMA, PRANDTL, TAU = 1.4, 0.71, 0.1
DEV = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------

def _case(name, op, etype, nx, ny, nz, P, viscous, flux, precision, beta=0.5, jitter=0.0, steps=1, cases=1):
    c = dict(op=op, etype=etype, nx=nx, ny=ny, nz=nz, P=P, viscous=viscous, flux=flux, precision=precision,
             beta=beta, jitter=jitter, steps=steps, cases=cases)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # A driver advancing a small 2D case by one step, its state exchanged
        # through torch: the smallest call, four stage launches.
        _case("vortex_quad_p3_step", "step", "quad", 32, 32, 0, 3, False, "rusanov", "fp64"),
        # Laminar flow around a cylinder (walls, far field, curved elements):
        # a few steps between two looks at the state.
        _case("cylinder_quad_p3_ns_step", "step", "cyl", 48, 96, 0, 3, True, "rusanov", "fp64", steps=4),
        # One residual of a 2D viscous run at high order in the mixed form on
        # a jittered mesh of odd size.
        _case("quad_p4_ns_mixed_residual", "residual", "quad", 147, 131, 0, 4, True, "roe", "mixed", jitter=0.1),
        # The triangle workload of the benchmark, a residual in the mixed form.
        _case("tri_p4_ns_mixed_residual", "residual", "tri", 128, 128, 0, 4, True, "roe", "mixed", jitter=0.15),
        # Triangles of another order, size and form, advanced in time.
        _case("tri_p3_ns_fp64_step", "step", "tri", 75, 75, 0, 3, True, "rusanov", "fp64", jitter=0.15, steps=2),
        # The benchmark's Taylor-Green residual: the largest call.
        _case("hex_p3_ns_fp64_residual", "residual", "hex", 64, 64, 64, 3, True, "roe", "fp64"),
        # A production Taylor-Green run in the mixed form: time steps.
        _case("hex_p3_ns_mixed_step", "step", "hex", 40, 40, 40, 3, True, "roe", "mixed", steps=2),
        # Inviscid flow on a ragged box at the reference's own flux.
        _case("hex_p2_euler_fp64_step", "step", "hex", 33, 29, 27, 2, False, "rusanov", "fp64", jitter=0.1, steps=2),
        # A higher odd point count per line, the reference's flux, jittered.
        _case("hex_p4_ns_fp64_residual", "residual", "hex", 23, 22, 21, 4, True, "rusanov", "fp64", jitter=0.1),
        # Sensitivities: one adjoint application on a 3D viscous case.
        _case("hex_p3_ns_vjp", "vjp", "hex", 24, 24, 24, 3, True, "roe", "fp64", jitter=0.1),
        # Shape and control gradients: the transpose of one time step of the
        # cylinder, as the reverse sweep calls it.
        _case("cylinder_quad_p3_step_vjp", "step_vjp", "cyl", 48, 96, 0, 3, True, "rusanov", "fp64"),
        # Many independent cases of mixed sizes and orders advanced together.
        _case("vortex_batch_mixed_step", "batch", "quad", 64, 64, 0, 5, False, "rusanov", "mixed", steps=10,
              cases=48),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["residual", "residual", "step", "step", "vjp", "step_vjp"])
    etype = rng.choice(["quad", "quad", "cyl", "tri", "tri", "hex", "hex", "hex"])
    viscous = etype == "cyl" or rng.random() < 0.75
    adjoint = op in ("vjp", "step_vjp")
    precision = "fp64" if adjoint else rng.choice(["fp64", "mixed"])
    flux = rng.choice(["rusanov", "roe"])
    beta = rng.choice([0.5, 0.5, 0.5, -0.5, 0.3]) if etype != "cyl" else 0.5
    jitter = rng.choice([0.0, 0.1]) if etype in ("quad", "hex") else (0.15 if etype == "tri" else 0.0)
    nz = 0
    if etype == "hex":
        P = rng.choice([1, 2, 3, 3] if adjoint else [1, 2, 3, 3, 4])
        most = {1: 32, 2: 30, 3: 28, 4: 20}[P]
        nx, ny, nz = (_log_int(rng, 5, 22 if adjoint else most) for _ in range(3))
    elif etype == "tri":
        P = rng.choice([1, 2, 3, 4, 5])
        nx = ny = _log_int(rng, 12, 60 if adjoint else 110)
    elif etype == "cyl":
        P = rng.choice([2, 3, 4])
        nx, ny = _log_int(rng, 12, 48), _log_int(rng, 24, 96)
    else:
        P = rng.choice([1, 2, 3, 4, 5])
        nx, ny = (_log_int(rng, 10, 64 if adjoint else 140) for _ in range(2))
    steps = rng.choice([1, 2, 3]) if op == "step" else 1
    return _case(None, op, etype, nx, ny, nz, P, viscous, flux, precision, beta, jitter, steps)


# ---------------------------------------------------------------------------
# meshes, parameters, points
# ---------------------------------------------------------------------------

BOX = {"quad": (-5.0, 5.0), "tri": (0.0, 1.0), "hex": (0.0, 2 * math.pi)}


def _mesh(case):
    e, nx, ny, nz = case["etype"], case["nx"], case["ny"], case["nz"]
    if e == "cyl":
        return meshgen.cylinder_omesh(nx, ny, wall_amp=(0.01, -0.005, 0.003, 0.002))
    if e == "tri":
        return meshgen.box_tris(nx, seed=2024, jitter=case["jitter"])
    m = meshgen.box_hexes(nx, ny, nz) if e == "hex" else meshgen.box_quads(nx, ny)
    if case["jitter"]:
        lo, hi = BOX[e]
        m = meshgen.jitter_interior(m, case["jitter"] * (hi - lo) / max(nx, ny, nz), 11)
    return m


def _physics(case):
    """Mach number, viscosity and time step (a fixed share of the stability limit)."""
    e, P = case["etype"], case["P"]
    c = math.sqrt(GAMMA)
    mach = {"quad": 0.5, "cyl": 0.2, "tri": 0.2, "hex": 0.1}[e]
    mu = mach * c / {"quad": 500.0, "cyl": 100.0, "tri": 1000.0, "hex": 1600.0}[e]
    if e == "cyl":
        h = 19.5 * 0.1 / (1.1 ** case["nx"] - 1.0)
        h = min(h, math.pi / case["ny"])
    else:
        lo, hi = BOX[e]
        h = (hi - lo) / max(case["nx"], case["ny"], case["nz"]) * (0.5 if e == "tri" else 1.0)
    dt = 0.1 * h / ((1.0 + mach) * c * (P + 1) ** 2)
    if case["viscous"]:
        dt = min(dt, 0.02 * h * h / (mu * (P + 1) ** 4))
    return mach, mu, dt


def _bounds(case):
    return {"WALL": "wall_ns_adi", "FARFIELD": "char"} if case["etype"] == "cyl" else {"PERIODIC": "periodic"}


def _new_solver(case):
    mach, mu, dt = _physics(case)
    p = make_params(case["P"], case["viscous"], gamma=GAMMA, prandtl=PRANDTL, mu=mu, ldg_b=case["beta"],
                    ldg_tau=TAU, V_fs=(mach * math.sqrt(GAMMA), 0.0, 0.0), dt=dt, fconv=case["flux"],
                    precision=case["precision"])
    s = FRSolver(_mesh(case), p, _bounds(case))
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    return s


_kept = collections.OrderedDict()


def _solver(case):
    """The case's solver.  A program sets its mesh up once and hands the
    solver one state after another, so states of a case share it; the two
    cases used last are kept."""
    key = repr(sorted((k, v) for k, v in case.items() if k not in ("name", "op", "steps")))
    if key not in _kept:
        while len(_kept) >= 2:
            _kept.popitem(last=False)[1].close()
        _kept[key] = _new_solver(case)
    _kept.move_to_end(key)
    return _kept[key]


def _gauss(N):
    return np.polynomial.legendre.leggauss(N)


def _lagrange(nodes, x):
    """[len(x), len(nodes)] Lagrange basis and its derivative at x."""
    n, val, der = len(nodes), np.ones((len(x), len(nodes))), np.zeros((len(x), len(nodes)))
    for m in range(n):
        for j in range(n):
            if j != m:
                val[:, m] *= (x - nodes[j]) / (nodes[m] - nodes[j])
                t = np.full(len(x), 1.0 / (nodes[m] - nodes[j]))
                for k in range(n):
                    if k not in (m, j):
                        t *= (x - nodes[k]) / (nodes[m] - nodes[k])
                der[:, m] += t
    return val, der


def _tables(etype, P, loc_tri=None):
    """Reference points in the library's orderings: solution points [S, D],
    flux points [Fp, D], their outward reference normals [Fp, D]."""
    N, x = P + 1, _gauss(P + 1)[0]
    if etype == "tri":
        spts = loc_tri
        r = 0.5 * math.sqrt(2.0)
        fpts = [(x[j], -1.0) for j in range(N)] + [(-x[j], x[j]) for j in range(N)] + [(-1.0, -x[j]) for j in range(N)]
        norm = [(0.0, -1.0)] * N + [(r, r)] * N + [(-1.0, 0.0)] * N
    elif etype == "hex":
        spts = [(x[k], x[j], x[i]) for i in range(N) for j in range(N) for k in range(N)]
        fpts, norm = [], []
        for face in range(6):
            for j in range(N):
                for k in range(N):
                    fpts.append([(x[k], x[j], -1.0), (-x[k], x[j], 1.0), (-1.0, x[k], x[j]), (1.0, -x[k], x[j]),
                                 (-x[k], -1.0, x[j]), (x[k], 1.0, x[j])][face])
                    n = [0.0, 0.0, 0.0]
                    n[(2, 2, 0, 0, 1, 1)[face]] = -1.0 if face % 2 == 0 else 1.0
                    norm.append(n)
    else:
        spts = [(x[j], x[i]) for i in range(N) for j in range(N)]
        fpts = [p for face in range(4) for p in
                [[(x[j], -1.0), (1.0, x[j]), (-x[j], 1.0), (-1.0, -x[j])][face] for j in range(N)]]
        norm = [n for n in [(0.0, -1.0), (1.0, 0.0), (0.0, 1.0), (-1.0, 0.0)] for _ in range(N)]
    return np.array(spts), np.array(fpts), np.array(norm)


GMSH_ORDER = {4: [0, 1, 3, 2], 9: [0, 2, 8, 6, 1, 5, 7, 3, 4], 8: [0, 1, 3, 2, 4, 5, 7, 6]}


def _shape(nn, loc):
    """Geometric shape functions [pts, nn] and derivatives [D, pts, nn] (gmsh node order)."""
    D = loc.shape[1]
    if nn == 3:
        v = np.stack([-(loc[:, 0] + loc[:, 1]) / 2, (1 + loc[:, 0]) / 2, (1 + loc[:, 1]) / 2], 1)
        return v, np.broadcast_to(np.array([[-0.5, 0.5, 0.0], [-0.5, 0.0, 0.5]])[:, None, :], (2, len(loc), 3)).copy()
    side = round(nn ** (1.0 / D))
    one = [_lagrange(np.linspace(-1, 1, side), loc[:, d]) for d in range(D)]
    val, der = np.empty((len(loc), nn)), np.empty((D, len(loc), nn))
    for g, st in enumerate(GMSH_ORDER[nn]):
        ix = [st // side ** d % side for d in range(D)]
        val[:, g] = np.prod([one[d][0][:, ix[d]] for d in range(D)], axis=0)
        for q in range(D):
            der[q][:, g] = np.prod([one[d][1 if d == q else 0][:, ix[d]] for d in range(D)], axis=0)
    return val, der


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=F64, device=DEV)


def _nodes(mesh):
    """Element node coordinates [nn, D, E]."""
    return _t(mesh.nodes[mesh.elements][:, :, :mesh.ndims].transpose(1, 2, 0))


@functools.lru_cache(maxsize=2)
def _tri_points(P):
    """The library's triangle solution points (where a state's values lie)."""
    from zefr_b200.solver import Plan
    plan = Plan(meshgen.box_tris(3), make_params(P), {"PERIODIC": "periodic"})
    return plan.get("loc_spts").reshape(-1, 2)


def _points(case, mesh):
    """Solution point coordinates [S, D, E]."""
    loc = _tables(case["etype"], case["P"], _tri_points(case["P"]) if case["etype"] == "tri" else None)[0]
    return torch.einsum("sn,nde->sde", _t(_shape(mesh.elements.shape[1], loc)[0]), _nodes(mesh))


# ---------------------------------------------------------------------------
# states
# ---------------------------------------------------------------------------

def _conserved(rho, vel, p):
    ke = sum(v * v for v in vel)
    return torch.stack([rho] + [rho * v for v in vel] + [p / (GAMMA - 1.0) + 0.5 * rho * ke], dim=1)


def _vortex(X, center, beta, mach):
    x, y = X[:, 0] - center[0], X[:, 1] - center[1]
    e = torch.exp(0.5 * (1.0 - x * x - y * y))
    T = 1.0 - (GAMMA - 1.0) * beta ** 2 / (8.0 * GAMMA * math.pi ** 2) * e * e
    rho = T ** (1.0 / (GAMMA - 1.0))
    b = beta / (2 * math.pi)
    return _conserved(rho, [mach * math.sqrt(GAMMA) - b * y * e, b * x * e], rho * T)


def _state(case, X, seed):
    """A flow on the points X [S, D, E] with the case's Mach number: vortices
    (inviscid quads), the stream around the cylinder with a near-wall layer
    and disturbances, or in a periodic box a field of random large modes with
    small point noise."""
    r = np.random.default_rng([seed, 7])
    mach, _, _ = _physics(case)
    U0, D = mach * math.sqrt(GAMMA), X.shape[1]
    if case["etype"] == "quad" and not case["viscous"]:
        return _vortex(X, r.uniform(-2, 2, 2), r.uniform(1, 5), mach)
    if case["etype"] == "cyl":
        R = torch.sqrt((X * X).sum(1))
        near = 1.0 - torch.exp(-4.0 * torch.clamp(R - 0.45, min=0.0))
        far = torch.exp(-0.5 * (R - 2.0) ** 2)
        ph = r.uniform(0, 2 * math.pi, 4)
        u = U0 * near * (1.0 + 0.05 * far * torch.sin(2 * X[:, 1] + ph[0]))
        v = 0.1 * U0 * near * far * torch.sin(3 * X[:, 0] + ph[1])
        p = 1.0 + 0.2 * U0 * U0 * far * torch.cos(X[:, 0] + X[:, 1] + ph[2])
        return _conserved(1.0 + 0.1 * U0 * U0 * far * torch.cos(2 * X[:, 0] + ph[3]), [u, v], p)
    lo, hi = BOX[case["etype"]]
    k0 = 2 * math.pi / (hi - lo)

    def field(amp, modes=3):
        f = torch.zeros_like(X[:, 0])
        for _ in range(modes):
            k = r.integers(-2, 3, D) * k0
            f += torch.sin(sum(float(k[d]) * X[:, d] for d in range(D)) + r.uniform(0, 2 * math.pi)) * r.normal()
        return amp * f / math.sqrt(modes)

    g = torch.Generator(device=X.device).manual_seed(seed)
    vel = [0.3 * U0 + field(U0) + 1e-3 * U0 * torch.randn(X[:, 0].shape, generator=g, device=X.device, dtype=F64)
           for _ in range(D)]
    return _conserved(1.0 + field(0.2 * U0 * U0), vel, 1.0 + field(0.3 * U0 * U0))


def _weight(shape, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 1)
    return torch.randn(shape, generator=g, device=DEV, dtype=F64)


def _batch_case_list(case):
    """Sizes and orders of the batch: fixed by the case (the flows by the seed)."""
    r = np.random.default_rng(4)
    out = []
    for _ in range(case["cases"]):
        n, P = int(r.integers(8, case["nx"] + 1)), int(r.integers(1, case["P"] + 1))
        out.append(dict(case, nx=n, ny=n, P=P))
    return out


def _batch_flow(sub, X, seed, i):
    r = np.random.default_rng([seed, i])
    return _vortex(X, r.uniform(-2, 2, 2), r.uniform(1, 5), r.uniform(0.2, 0.8))


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    if case["op"] == "batch":
        solvers = []
        for i, sub in enumerate(_batch_case_list(case)):
            s = _new_solver(sub)
            s.set_state(_batch_flow(sub, _points(sub, _mesh(sub)), seed, i))
            solvers.append(s)
        return {"case": case, "solvers": solvers, "batch": Batch(solvers),
                "out": [torch.empty(s.state_shape, dtype=F64, device=DEV) for s in solvers]}
    s = _solver(case)
    U = _state(case, _points(case, _mesh(case)), seed).contiguous()
    st = {"case": case, "solver": s, "U": U, "out": torch.empty_like(U)}
    if case["op"] in ("vjp", "step_vjp"):
        st["lam"] = _weight(s.state_shape, seed)
    return st


def run(st):
    case = st["case"]
    op = case["op"]
    if op == "batch":
        st["batch"].step(case["steps"])
        st["batch"].synchronize()
        for s, out in zip(st["solvers"], st["out"]):
            s.get_state_device(out)
        return st["out"]
    s = st["solver"]
    if op == "step_vjp":
        pbar = np.zeros(5)
        return {"U": s.rk_step_vjp(st["U"], st["lam"], pbar), "freestream": pbar}
    s.set_state(st["U"])
    if op == "vjp":
        return s.vjp(st["lam"])
    if op == "residual":
        s.compute_residual(0)
        s.get_residual_device(st["out"])
    else:
        s.step(case["steps"])
        s.get_state_device(st["out"])
    return st["out"]


# ---------------------------------------------------------------------------
# work and tolerance
# ---------------------------------------------------------------------------

def _sizes(case):
    P, N, e = case["P"], case["P"] + 1, case["etype"]
    if e == "hex":
        return 3, N ** 3, 6 * N * N, case["nx"] * case["ny"] * case["nz"]
    if e == "tri":
        return 2, N * (N + 1) // 2, 3 * N, 2 * case["nx"] * case["nx"]
    return 2, N * N, 4 * N, case["nx"] * case["ny"]


def work(case):
    if case["op"] == "batch":
        w = [work(dict(c, op="step")) for c in _batch_case_list(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    D, S, Fp, E = _sizes(case)
    V, N = D + 2, case["P"] + 1
    w = 8 if case["precision"] == "fp64" else 4
    geo = E * S * (D * D + 1) * w + E * Fp * ((D + 2) * w / 2 + 5)  # metrics, normals, connectivity
    pts = E * S * V
    # operations of one residual: extrapolation, flux transform and divergence,
    # surface terms, common flux (once per point pair); viscous: gradient with
    # its transform, its traces on one side
    dense = case["etype"] == "tri"
    line_e, line_d = (S, S) if dense else (N, N)
    surf = Fp if dense else 2 * D
    f = 2 * line_e * Fp * V + (2 * D * line_d + 2 * D * D + 2 * surf) * S * V + 20 * D * S + 60 * D * Fp / 2
    if case["viscous"]:
        f += (2 * D * line_d + 2 * surf + 2 * D * D) * S * V + D * line_e * Fp * V + 30 * D * S + 30 * D * Fp / 2
    f *= E
    op = case["op"]
    if op == "residual":  # state in, residual out, as the caller's FP64 arrays
        return {"bytes": 16 * pts + geo, "flops": f}
    if op == "step":      # per stage the state and a running sum, in and out
        n = 4 * case["steps"]
        return {"bytes": 16 * pts + n * (4 * pts * w + geo), "flops": n * (f + 6 * pts)}
    if op == "vjp":       # state and weight in, adjoint out; about two residuals' operations
        return {"bytes": 24 * pts + geo, "flops": 2 * f}
    # four stages forward (their states and residuals kept) and four back
    return {"bytes": 24 * pts + 8 * (4 * pts * w + geo), "flops": 12 * f}


def tolerance(case):
    """About four times the largest difference seen between the library's
    outputs and the 64-bit values of ``exact`` over the listed and drawn cases.
    A residual loses digits where it is a small difference of large fluxes, at
    the low Mach number of the hexahedral cases above all; an advanced state
    hides all but its last digits."""
    low = case["etype"] == "hex"
    if case["precision"] == "fp64":
        if case["op"] == "step":
            return {"rel": 4e-15, "max": 1e-13}
        if case["op"] == "residual":
            return {"rel": 4e-11, "max": 2e-9}
        return {"rel": 1e-12, "max": 1e-10}
    if case["op"] == "residual":
        return {"rel": 2e-3, "max": 0.1} if low else {"rel": 6e-4, "max": 0.03}
    return {"rel": 2e-8, "max": 1e-6}


# ---------------------------------------------------------------------------
# the same outputs in plain 64-bit torch: dense operators, gathered faces
# ---------------------------------------------------------------------------

def _tri_basis(P, pts):
    """Legendre products of total degree <= P at pts, and derivatives."""
    L = [np.polynomial.legendre.Legendre.basis(i) for i in range(P + 1)]
    idx = [(i, k - i) for k in range(P + 1) for i in range(k + 1)]
    x, y = pts[:, 0], pts[:, 1]
    return (np.stack([L[i](x) * L[j](y) for i, j in idx], 1),
            np.stack([L[i].deriv()(x) * L[j](y) for i, j in idx], 1),
            np.stack([L[i](x) * L[j].deriv()(y) for i, j in idx], 1))


def _operators(case):
    """Dense E [Fp, S], G [D, S, S], Gf [D, S, Fp], Dv [D, S, S], Df [S, Fp]."""
    e, P = case["etype"], case["P"]
    N = P + 1
    sp, fp, nr = _tables(e, P, _tri_points(P) if e == "tri" else None)
    D, S, Fp = sp.shape[1], len(sp), len(fp)
    x, w = _gauss(N)
    if e == "tri":
        V, Vx, Vy = _tri_basis(P, sp)
        Vf = _tri_basis(P, fp)[0]
        E = Vf @ np.linalg.inv(V)
        qx, qw = _gauss(P + 2)
        a, b = np.meshgrid(qx, qx)
        q = np.stack([((1 + a) * (1 - b) / 2 - 1).ravel(), b.ravel()], 1)
        Q = _tri_basis(P, q)[0]
        gram = Q.T @ (Q * (np.outer(qw, qw) * (1 - b) / 2).ravel()[:, None])
        Df = V @ np.linalg.solve(gram, Vf.T) * np.tile(w, 3)[None, :]
        Gf = np.stack([Df * nr[:, d] for d in range(D)])
        G = np.stack([W @ np.linalg.inv(V) for W in (Vx, Vy)]) - np.einsum("dsf,ft->dst", Gf, E)
        # the reference's triangle divergence holds the surface part only
        Dv = -np.stack([Df * nr[:, d] @ E for d in range(D)])
        return E, G, Gf, Dv, Df
    ext = np.concatenate([[-1.0], x, [1.0]])
    ends = _lagrange(x, np.array([-1.0, 1.0]))[0]
    der = _lagrange(ext, x)[1]
    E, G, Gf = np.zeros((Fp, S)), np.zeros((D, S, S)), np.zeros((D, S, Fp))
    for f in range(Fp):
        d = int(np.argmax(np.abs(nr[f])))
        side = int(nr[f][d] > 0)
        others = [q for q in range(D) if q != d]
        for s in np.nonzero(np.all(np.abs(sp[:, others] - fp[f][others]) < 1e-9, axis=1))[0]:
            i = int(np.argmin(np.abs(x - sp[s][d])))
            E[f, s] = ends[side, i]
            Gf[d, s, f] = der[i, N + 1 if side else 0]
    for d in range(D):
        others = [q for q in range(D) if q != d]
        for s in range(S):
            i = int(np.argmin(np.abs(x - sp[s][d])))
            for t in np.nonzero(np.all(np.abs(sp[:, others] - sp[s][others]) < 1e-9, axis=1))[0]:
                G[d, s, t] = der[i, int(np.argmin(np.abs(x - sp[t][d]))) + 1]
    return E, G, Gf, G.copy(), np.einsum("dsf,fd->sf", Gf, nr)


def _adjugate(J):
    """J [D (reference), P, D (physical), E] -> |J|-scaled inverse transposed: adj[d1][d2] and |J|."""
    if J.shape[0] == 2:
        return torch.stack([torch.stack([J[1, :, 1], -J[1, :, 0]], 1), torch.stack([-J[0, :, 1], J[0, :, 0]], 1)]), \
            J[0, :, 0] * J[1, :, 1] - J[0, :, 1] * J[1, :, 0]
    rows = [torch.linalg.cross(J[(d + 1) % 3], J[(d + 2) % 3], dim=1) for d in range(3)]
    return torch.stack(rows), (J[0] * rows[0]).sum(1)


FACES = {"quad": [[0, 1], [1, 2], [2, 3], [3, 0]], "cyl": [[0, 1], [1, 2], [2, 3], [3, 0]],
         "tri": [[0, 1], [1, 2], [2, 0]],
         "hex": [[0, 1, 2, 3], [5, 4, 7, 6], [0, 3, 7, 4], [2, 1, 5, 6], [1, 0, 4, 5], [3, 2, 6, 7]]}


def _face_pairs(case, mesh):
    """(left, right) element-face numbers e * nfaces + n of interior and
    periodic faces (left: the element met first), and those on a boundary."""
    ids = np.arange(mesh.nodes.shape[0])
    if case["etype"] != "cyl":  # periodic images share one number
        n = [case["nx"], case["ny"], max(case["nz"], 0)][:mesh.ndims]
        c, ids, left = [], 0, np.arange(mesh.nodes.shape[0])
        for k in n:
            c.append(left % (k + 1) % k)
            left = left // (k + 1)
        for k, q in zip(n[::-1], c[::-1]):
            ids = ids * k + q
    keys = np.sort(ids[mesh.elements][:, np.array(FACES[case["etype"]])], axis=2)
    keys = keys.reshape(-1, keys.shape[2])
    order = np.lexsort(keys.T[::-1])
    same = np.all(keys[order[1:]] == keys[order[:-1]], axis=1)
    L, R = order[:-1][same], order[1:][same]
    alone = np.setdiff1d(np.arange(len(keys)), np.concatenate([L, R]))
    return np.minimum(L, R), np.maximum(L, R), alone


class _Exact:
    """The discretisation in dense form: state [S, V, E], flux points flat [Fp * E]."""

    def __init__(self, case):
        mesh = _mesh(case)
        self.visc, self.roe, self.beta = case["viscous"], case["flux"] == "roe", case["beta"]
        self.mach, self.mu, self.dt = _physics(case)
        sp, fp, nr = _tables(case["etype"], case["P"], _tri_points(case["P"]) if case["etype"] == "tri" else None)
        self.D, self.S, self.Fp, self.E = sp.shape[1], len(sp), len(fp), mesh.elements.shape[0]
        self.oE, self.oG, self.oGf, self.oD, self.oDf = (_t(a) for a in _operators(case))
        X = _nodes(mesh)
        nn = X.shape[0]
        self.adj, self.det = _adjugate(torch.einsum("dpn,nxe->dpxe", _t(_shape(nn, sp)[1]), X))
        vf, df = _shape(nn, fp)
        fadj = _adjugate(torch.einsum("dpn,nxe->dpxe", _t(df), X))[0]
        nrm = torch.einsum("dpxe,pd->pxe", fadj, _t(nr))
        del fadj
        self.dA = torch.sqrt((nrm * nrm).sum(1)).reshape(-1)
        nrm = (nrm / self.dA.reshape(self.Fp, 1, self.E)).permute(1, 0, 2).reshape(self.D, -1)
        xf = torch.einsum("pn,nxe->pxe", _t(vf), X)
        # faces: flux points of both sides paired by place relative to the face's centre
        nf = len(FACES[case["etype"]])
        k = self.Fp // nf
        L, R, B = _face_pairs(case, mesh)

        def points(face):
            face = torch.as_tensor(face, device=DEV)
            return ((face % nf)[:, None] * k + torch.arange(k, device=DEV)) * self.E + (face // nf)[:, None]

        def place(pt):
            x = xf[pt // self.E, :, pt % self.E]
            return x - x.mean(1, keepdim=True)

        l, r = points(L), points(R)
        match = torch.empty_like(l)
        for a in range(0, len(l), 1 << 17):
            xl, xr = place(l[a:a + (1 << 17)]), place(r[a:a + (1 << 17)])
            match[a:a + (1 << 17)] = (xl[:, :, None] - xr[:, None]).abs().amax(3).argmin(2)
        r = torch.gather(r, 1, match)
        self.l, self.r, self.b = l.reshape(-1), r.reshape(-1), points(B).reshape(-1)
        self.n, self.nb = nrm[:, self.l], nrm[:, self.b]
        if len(B):
            xb = xf[self.b // self.E, :, self.b % self.E]
            self.wall = torch.sqrt((xb * xb).sum(1)) < 5.0

    # fluxes: states [V, ...], gradients [V, D, ...], normals [D, ...]
    def prim(self, U):
        vel = U[1:-1] / U[0]
        p = (GAMMA - 1.0) * (U[-1] - 0.5 * (U[1:-1] * vel).sum(0))
        return vel, p

    def normal_flux(self, U, n):
        vel, p = self.prim(U)
        vn = (vel * n).sum(0)
        return torch.cat([(U[0] * vn)[None], U[1:-1] * vn + p * n, ((U[-1] + p) * vn)[None]]), vn, p

    def riemann(self, UL, UR, n):
        FL, vL, pL = self.normal_flux(UL, n)
        FR, vR, pR = self.normal_flux(UR, n)
        if not self.roe:
            lam = torch.maximum(vL.abs() + torch.sqrt(GAMMA * pL / UL[0]), vR.abs() + torch.sqrt(GAMMA * pR / UR[0]))
            return 0.5 * (FL + FR) - 0.5 * lam * (UR - UL)
        # Roe averages with Harten's fix below a tenth of the largest wave speed
        sL, sR = torch.sqrt(UL[0]), torch.sqrt(UR[0])
        velL, velR = UL[1:-1] / UL[0], UR[1:-1] / UR[0]
        u = (sL * velL + sR * velR) / (sL + sR)
        H = (sL * (UL[-1] + pL) / UL[0] + sR * (UR[-1] + pR) / UR[0]) / (sL + sR)
        q2, un = (u * u).sum(0), (u * n).sum(0)
        a2 = (GAMMA - 1.0) * (H - 0.5 * q2)
        a, rho = torch.sqrt(a2), sL * sR
        dp, dr, dn = pR - pL, UR[0] - UL[0], vR - vL
        delta = 0.1 * (un.abs() + a)

        def fix(x):
            x = x.abs()
            return torch.where(x < delta, (x * x + delta * delta) / (2 * delta), x)

        w1 = fix(un - a) * (dp - rho * a * dn) / (2 * a2)
        w3 = fix(un + a) * (dp + rho * a * dn) / (2 * a2)
        l2, s = fix(un), dr - dp / a2
        dt = (velR - velL) - dn * n
        diss = torch.cat([(w1 + l2 * s + w3)[None], w1 * (u - a * n) + l2 * (s * u + rho * dt) + w3 * (u + a * n),
                          (w1 * (H - a * un) + l2 * (0.5 * s * q2 + rho * (u * dt).sum(0)) + w3 * (H + a * un))[None]])
        return 0.5 * (FL + FR) - 0.5 * diss

    def viscous(self, U, dU):
        """Minus the viscous flux [V, D, ...]."""
        vel = U[1:-1] / U[0]
        g = (dU[1:-1] - dU[0] * vel[:, None]) / U[0]              # g[i, j] = d u_i / d x_j
        e = U[-1] / U[0] - 0.5 * (vel * vel).sum(0)
        de = (dU[-1] - dU[0] * U[-1] / U[0]) / U[0] - (vel[:, None] * g).sum(0)
        div = sum(g[i, i] for i in range(self.D))
        tau = self.mu * (g + g.transpose(0, 1))
        tau = torch.stack([torch.stack([tau[i, j] - (2.0 / 3.0 * self.mu * div if i == j else 0.0)
                                        for j in range(self.D)]) for i in range(self.D)])
        heat = self.mu * GAMMA / PRANDTL * de
        return -torch.cat([torch.zeros_like(dU[:1]), tau, ((vel[:, None] * tau).sum(0) + heat)[None]])

    def ghost(self, U, fs):
        """Riemann and viscous states beyond the boundary points: adiabatic
        no-slip walls, the characteristic far field elsewhere."""
        rho_fs, V_fs, p_fs = fs[0], fs[1:1 + self.D], fs[4]
        n, g1 = self.nb, GAMMA - 1.0
        vel, p = self.prim(U)
        vn, vf = (vel * n).sum(0), (V_fs[:, None] * n).sum(0)
        cL, cR = torch.sqrt(GAMMA * p / U[0]), torch.sqrt(GAMMA * p_fs / rho_fs)
        hi, lo = vn + 2 / g1 * cL, vf - 2 / g1 * cR                # subsonic far field
        c, un = 0.25 * g1 * (hi - lo), 0.5 * (hi + lo)
        inflow = vn < 0
        s = torch.where(inflow, rho_fs ** GAMMA / p_fs, U[0] ** GAMMA / p)
        v = torch.where(inflow, V_fs[:, None] + (un - vf) * n, vel + (un - vn) * n)
        rho = (c * c / GAMMA * s) ** (1.0 / g1)
        far = torch.cat([rho[None], rho * v, (rho * c * c / GAMMA / g1 + 0.5 * rho * (v * v).sum(0))[None]])
        still = torch.cat([U[:1], torch.zeros_like(U[1:-1]), (U[-1] - 0.5 * U[0] * (vel * vel).sum(0))[None]])
        turned = torch.cat([U[:1], -U[1:-1], U[-1:]])
        return torch.where(self.wall, turned, far), torch.where(self.wall, still, far)

    def residual(self, U, fs=None):
        D, S, V, E, Fp = self.D, self.S, U.shape[1], self.E, self.Fp
        l, r, b = self.l, self.r, self.b
        Uf = torch.einsum("fs,sve->vfe", self.oE, U).reshape(V, Fp * E)
        UL, UR, Ub = Uf[:, l], Uf[:, r], Uf[:, b]
        if fs is None:
            fs = _t([1.0, self.mach * math.sqrt(GAMMA), 0.0, 0.0, 1.0])
        Ug, UB = self.ghost(Ub, fs) if len(b) else (Ub, Ub)
        Fi = self.riemann(UL, UR, self.n)
        Fb = self.riemann(Ub, Ug, self.nb)
        Us = U.transpose(0, 1)                                        # [V, S, E]
        vel, p = self.prim(Us)
        F = Us[:, None] * vel[None]
        F = F + torch.cat([torch.zeros_like(F[:1]), p * torch.eye(D, dtype=F64, device=DEV)[:, :, None, None],
                           (p * vel)[None]])
        if self.visc:
            beta = self.beta
            uc = 0.5 * (UL + UR) - beta * (UL - UR)
            C = torch.empty_like(Uf).index_copy(1, l, uc).index_copy(1, r, uc).index_copy(1, b, UB)
            dR = torch.einsum("dst,tve->dvse", self.oG, U) + \
                torch.einsum("dsf,vfe->dvse", self.oGf, C.reshape(V, Fp, E))
            dU = torch.einsum("dvse,dsxe->vxse", dR, self.adj) / self.det
            del dR
            F = F + self.viscous(Us, dU)
            dF = torch.einsum("fs,vxse->vxfe", self.oE, dU).reshape(V, D, Fp * E)
            del dU
            FL = (self.viscous(UL, dF[:, :, l]) * self.n).sum(1)
            FR = (self.viscous(UR, dF[:, :, r]) * self.n).sum(1)
            Fi = Fi + (0.5 + beta) * FL + (0.5 - beta) * FR + TAU * (UL - UR)
            if len(b):  # no heat through an adiabatic wall
                db, vb = dF[:, :, b], Ub[1:-1] / Ub[0]
                gv = (db[1:-1] - db[0] * vb[:, None]) / Ub[0]
                dT = db[-1] - db[0] * Ub[-1] / Ub[0] - Ub[0] * (vb[:, None] * gv).sum(0)
                dTn = torch.where(self.wall, (dT * self.nb).sum(0), 0.0)
                db = torch.cat([db[:-1], (db[-1] - dTn * self.nb)[None]])
                Fb = Fb + (self.viscous(UB, db) * self.nb).sum(1) + TAU * (Ub - UB)
            del dF
        Ft = torch.einsum("vxse,dsxe->dsve", F, self.adj)
        C = torch.empty_like(Uf).index_copy(1, l, Fi * self.dA[l]).index_copy(1, r, -Fi * self.dA[r])
        C = C.index_copy(1, b, Fb * self.dA[b])
        return torch.einsum("dst,dtve->sve", self.oD, Ft) + torch.einsum("sf,vfe->sve", self.oDf, C.reshape(V, Fp, E))

    def step(self, U, fs=None):
        c = self.dt / self.det[:, None, :]
        k1 = self.residual(U, fs)
        k2 = self.residual(U - 0.5 * c * k1, fs)
        k3 = self.residual(U - 0.5 * c * k2, fs)
        k4 = self.residual(U - c * k3, fs)
        return U - c / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + k4)


def exact(case, seed):
    op = case["op"]
    if op == "batch":
        out = []
        for i, sub in enumerate(_batch_case_list(case)):
            ex, U = _Exact(sub), _batch_flow(sub, _points(sub, _mesh(sub)), seed, i)
            for _ in range(case["steps"]):
                U = ex.step(U)
            out.append(U)
        return out
    ex = _Exact(case)
    U = _state(case, _points(case, _mesh(case)), seed).contiguous()
    if op == "residual":
        return ex.residual(U)
    if op == "step":
        for _ in range(case["steps"]):
            U = ex.step(U)
        return U
    lam = _weight(U.shape, seed)
    fs = _t([1.0, ex.mach * math.sqrt(GAMMA), 0.0, 0.0, 1.0]).requires_grad_()
    U.requires_grad_()
    if op == "vjp":
        return torch.autograd.grad(ex.residual(U, fs), U, lam)[0]
    gU, gf = torch.autograd.grad(ex.step(U, fs), [U, fs], lam, allow_unused=True)
    return {"U": gU, "freestream": None if gf is None else gf.cpu().numpy()}
