"""Hexahedral kernels whose columns are shared by several threads, over every
order, one ragged tile to several, and both LDG forms, against the numpy
oracle."""
import numpy as np
import pytest

from oracle import dfr_numpy as O
from zefr_b200 import meshgen
from zefr_b200.solver import FRSolver, make_params

pytestmark = pytest.mark.gpu

PHYS = dict(gamma=1.4, prandtl=0.71, mu=2e-3, fix_vis=1, rus_k=0.0, ldg_tau=0.1, rho_fs=1.0, P_fs=1.0, T_wall=0.0,
            R_ref=0.0, rt=0.0, c_sth=0.0, **{f"V_{w}{d}": 0.0 for w in ("fs", "wall") for d in range(3)})


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("mixed", 1e-4)])
@pytest.mark.parametrize("viscous,beta,fconv", [(False, 0.5, "rusanov"), (True, 0.5, "roe"), (True, -0.5, "rusanov"),
                                                (True, 0.3, "rusanov")])
@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [(3, 3, 3), (5, 3, 4)])
def test_residual_and_step(n, order, viscous, beta, fconv, precision, tol):
    """FP64: rounding of a few hundred operations.  Mixed: 2^-24 in values and
    products of order one against residuals of order 1e-2 and more."""
    mesh = meshgen.jitter_interior(meshgen.box_hexes(*n), 0.1, 3)
    p = make_params(order, viscous, gamma=1.4, prandtl=0.71, mu=2e-3, ldg_b=beta, ldg_tau=0.1, fconv=fconv,
                    precision=precision, dt=1e-3)
    s = FRSolver(mesh, p, {"PERIODIC": "periodic"})
    st = O.Setup.from_arrays(3, s.nspts, s.info.nfpts, s.neles, s.plan.get)
    rng = np.random.default_rng(order)
    X = s.plan.get("coord_spts").reshape(s.nspts, 3, s.neles)
    U = np.ones(s.state_shape)
    for v in range(5):
        k = rng.integers(1, 3, 3)
        U[:, v] = (0.0 if 0 < v < 4 else 1.0 + 1.5 * (v == 4)) + 0.1 * np.sin(X[:, 0] * k[0] + v) * np.cos(
            X[:, 1] * k[1]) * np.cos(X[:, 2] * k[2] + 1)
    d = dict(PHYS, ldg_b=beta)
    want = O.residual(st, U, d, viscous, fconv)
    got = s.residual(U)
    scale = np.abs(want).max(axis=(0, 2))
    assert (np.abs(got - want).max(axis=(0, 2)) <= tol * scale).all()
    # the RK stages (update and next traces) end where residual by residual ends
    s.step(1)
    Us, regs = U, []
    for a in (0.5, 0.5, 1.0, None):
        regs.append(O.residual(st, Us, d, viscous, fconv))
        if a is not None:
            Us = U - a * 1e-3 / st.jaco_det[:, None] * regs[-1]
    Un = U - 1e-3 / st.jaco_det[:, None] * (regs[0] + 2 * regs[1] + 2 * regs[2] + regs[3]) / 6
    step_tol = 1e-13 if precision == "fp64" else 1e-6
    assert np.abs(s.get_state() - Un).max() <= step_tol


@pytest.mark.parametrize("n,order,viscous,beta", [((18, 17, 17), 1, True, 0.5), ((18, 17, 17), 1, True, 0.3),
                                                  ((16, 16, 16), 2, False, 0.5)])
def test_shapes_chosen_by_mesh_size(n, order, viscous, beta):
    """FP64 P1 gradient kernel past the 592 tiles that four CTAs per SM hold (the
    meshes above stay below), P2 Euler kernel between three and four CTAs per SM
    (512 tiles); tolerances as above."""
    test_residual_and_step(n, order, viscous, beta, "rusanov", "fp64", 1e-12)
