"""Quadrilateral and triangle kernels over every order (one thread per point,
so thread counts and remainders change with the order), one ragged tile to
more tiles than resident CTAs, and each LDG form, against the numpy oracle."""
import numpy as np
import pytest

from oracle import dfr_numpy as O
from zefr_b200 import meshgen
from zefr_b200.solver import FRSolver, make_params

pytestmark = pytest.mark.gpu

PHYS = dict(gamma=1.4, prandtl=0.71, mu=2e-3, fix_vis=1, rus_k=0.0, ldg_tau=0.1, rho_fs=1.0, P_fs=1.0, T_wall=0.0,
            R_ref=0.0, rt=0.0, c_sth=0.0, **{f"V_{w}{d}": 0.0 for w in ("fs", "wall") for d in range(3)})
FORMS = [(False, 0.5, "rusanov"), (True, 0.5, "roe"), (True, -0.5, "rusanov"), (True, 0.3, "roe")]
QUADS = [("quad", n, p) for p in (1, 2, 3, 4, 5) for n in ((3, 3), (7, 5))]
TRIS = [("tri", n, p) for p in (1, 2, 3, 4, 5, 6, 7, 8) for n in ((3,), (5,))]


def _state(s):
    X = s.plan.get("coord_spts").reshape(s.nspts, 2, s.neles)
    U = np.ones(s.state_shape)
    for v in range(4):
        U[:, v] = (0.0 if v in (1, 2) else 1.0 + 1.5 * (v == 3)) + 0.1 * np.sin(2 * np.pi * X[:, 0] + v) * np.cos(
            2 * np.pi * X[:, 1] + 1)
    # jumps at the faces: the reference's triangle residual is their lift alone
    return U + 0.02 * np.random.default_rng(0).uniform(-1.0, 1.0, U.shape)


def _case(kind, n, order, viscous, beta, fconv, precision, dt):
    mesh = (meshgen.jitter_interior(meshgen.box_quads(*n, 0.0, 1.0, 0.0, 1.0), 0.1 / max(n), 3) if kind == "quad"
            else meshgen.box_tris(*n, jitter=0.1))
    p = make_params(order, viscous, gamma=1.4, prandtl=0.71, mu=2e-3, ldg_b=beta, ldg_tau=0.1, fconv=fconv,
                    precision=precision, dt=dt)
    return FRSolver(mesh, p, {"PERIODIC": "periodic"})


@pytest.mark.parametrize("precision,tol", [("fp64", 2e-12), ("mixed", 1e-4)])
@pytest.mark.parametrize("viscous,beta,fconv", FORMS)
@pytest.mark.parametrize("kind,n,order", QUADS + TRIS)
def test_residual_and_step(kind, n, order, viscous, beta, fconv, precision, tol):
    """FP64: rounding of a few hundred operations, dense triangle rows of up to
    90 terms.  Mixed: 2^-24 in values and products of order one against
    residuals of order 1e-2 and more."""
    dt = 1e-4
    s = _case(kind, n, order, viscous, beta, fconv, precision, dt)
    st = O.Setup.from_arrays(2, s.nspts, s.info.nfpts, s.neles, s.plan.get)
    U, d = _state(s), dict(PHYS, ldg_b=beta)
    want = O.residual(st, U, d, viscous, fconv)
    got = s.residual(U)
    scale = np.abs(want).max(axis=(0, 2))
    assert (np.abs(got - want).max(axis=(0, 2)) <= tol * scale).all()
    s.step(1)
    Us, regs = U, []
    for a in (0.5, 0.5, 1.0, None):
        regs.append(O.residual(st, Us, d, viscous, fconv))
        if a is not None:
            Us = U - a * dt / st.jaco_det[:, None] * regs[-1]
    Un = U - dt / st.jaco_det[:, None] * (regs[0] + 2 * regs[1] + 2 * regs[2] + regs[3]) / 6
    assert np.abs(s.get_state() - Un).max() <= (1e-13 if precision == "fp64" else 1e-6)


@pytest.mark.parametrize("precision,tol", [("fp64", 2e-12), ("mixed", 1e-4)])
@pytest.mark.parametrize("beta,fconv", [(0.5, "roe"), (0.3, "rusanov")])
def test_quads_p5_of_more_tiles_than_sms(beta, fconv, precision, tol):
    """154 tiles: the FP64 face kernel takes its two-CTA form past 148
    (tolerances as in test_residual_and_step)."""
    test_residual_and_step("quad", (41, 30), 5, True, beta, fconv, precision, tol)


@pytest.mark.parametrize("kind,n", [("quad", (123, 97)), ("tri", (91,))])
def test_many_tiles_repeat_the_few(kind, n):
    """More tiles than fit the GPU at once: a uniform state stays uniform and
    the residual of a state does not depend on the run."""
    s = _case(kind, n, 3, True, 0.5, "rusanov", "fp64", 1e-4)
    U = _state(s)
    R = s.residual(U)
    assert np.array_equal(R, s.residual(U))
    C = np.broadcast_to(np.array([1.0, 0.3, -0.2, 2.7])[None, :, None], s.state_shape)
    assert np.abs(s.residual(C)).max() < 1e-12


# Meshes (box_tris(n): 2 n^2 elements, 8 to a tile) of more tiles than the
# GPU holds CTAs of any triangle kernel of that order and form (148 SMs times
# the most CTAs per SM: 20, 13, 13, 3 of the FP32 gradient and Euler kernels at
# P1, P2, P3, P8, 16, 16, 4 of the extrapolation from P2 on; FP64 8, 5, 5, 1):
# every CTA walks on to another tile, in FP64 to several.  P1 n 125 and P2 n 184
# are also where the extrapolation takes its form for large meshes.
MANY = [("fp64", 1, 125), ("fp64", 2, 100), ("mixed", 2, 100), ("fp64", 2, 184), ("mixed", 2, 184),
        ("fp64", 3, 100), ("fp64", 8, 45), ("mixed", 1, 125), ("mixed", 3, 105), ("mixed", 8, 52)]


@pytest.mark.parametrize("viscous,beta,fconv", [(False, 0.5, "roe"), (True, 0.5, "rusanov"), (True, 0.3, "roe")])
@pytest.mark.parametrize("precision,order,n", MANY)
def test_triangles_of_more_tiles_than_resident_ctas(precision, order, n, viscous, beta, fconv):
    """Residual and step against the oracle on a state that differs from tile
    to tile (random jumps), so a CTA that read what its last tile left behind
    would show.  Tolerances as in test_residual_and_step; the step adds a
    multiple of dt / h of the residual's error, both small."""
    dt = 1e-6
    s = _case("tri", (n,), order, viscous, beta, fconv, precision, dt)
    st = O.Setup.from_arrays(2, s.nspts, s.info.nfpts, s.neles, s.plan.get)
    U, d = _state(s), dict(PHYS, ldg_b=beta)
    tol = 2e-12 if precision == "fp64" else 1e-4
    want = O.residual(st, U, d, viscous, fconv)
    scale = np.abs(want).max(axis=(0, 2))
    assert (np.abs(s.residual(U) - want).max(axis=(0, 2)) <= tol * scale).all()
    s.set_state(U)
    s.step(1)
    Us, regs = U, [want]
    for a in (0.5, 0.5, 1.0):
        Us = U - a * dt / st.jaco_det[:, None] * regs[-1]
        regs.append(O.residual(st, Us, d, viscous, fconv))
    Un = U - dt / st.jaco_det[:, None] * (regs[0] + 2 * regs[1] + 2 * regs[2] + regs[3]) / 6
    moved = np.abs(Un - U).max()
    err = np.abs(s.get_state() - Un).max()
    assert err <= (1e-13 + tol * moved if precision == "fp64" else 1e-6)
    s.close()


# every boundary kind through the two-dimensional kernels
WALLS = [("wall_ns_adi", True), ("wall_ns_iso", True), ("char", True), ("char", False), ("wall_slip", False)]


@pytest.mark.parametrize("precision,tol", [("fp64", 2e-12), ("mixed", 1e-4)])
@pytest.mark.parametrize("bc,viscous", WALLS)
@pytest.mark.parametrize("kind,n,order", [("quad", (5, 4), p) for p in (1, 2, 3, 4, 5)] +
                         [("tri", (4,), p) for p in (1, 2, 3, 4, 5, 6, 7, 8)])
def test_boundaries(kind, n, order, bc, viscous, precision, tol):
    """A box whose four sides are one boundary, at every order, against the
    oracle (tolerances as in test_residual_and_step)."""
    mesh = (meshgen.jitter_interior(meshgen.box_quads(*n, 0.0, 1.0, 0.0, 1.0, bnd="SIDE"), 0.02, 3) if kind == "quad"
            else meshgen.box_tris(*n, jitter=0.1, bnd="SIDE"))
    p = make_params(order, viscous, gamma=1.4, prandtl=0.71, mu=2e-3, ldg_b=0.5, ldg_tau=0.1, precision=precision,
                    V_fs=(0.3, 0.1, 0.0), rho_fs=1.0, P_fs=1.0, T_wall=1.0, R_ref=1.0)
    s = FRSolver(mesh, p, {"SIDE": bc})
    st = O.Setup.from_arrays(2, s.nspts, s.info.nfpts, s.neles, s.plan.get)
    U = _state(s)
    d = dict(PHYS, ldg_b=0.5, V_fs0=0.3, V_fs1=0.1, T_wall=1.0, R_ref=1.0)
    want = O.residual(st, U, d, viscous)
    scale = np.abs(want).max(axis=(0, 2))
    assert (np.abs(s.residual(U) - want).max(axis=(0, 2)) <= tol * scale).all()
    s.close()
