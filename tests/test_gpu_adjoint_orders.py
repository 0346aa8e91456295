"""Viscous adjoint of quadrilaterals at every order: lam . (dR/dU) v by central
differences of the FP64 residual against (dR/dU)^T lam . v, and the same bits
twice (from P4 on a tile has more solution than flux points)."""
import numpy as np
import pytest

from zefr_b200 import meshgen
from zefr_b200.solver import FRSolver, make_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bounds", ["periodic", "walls"])
@pytest.mark.parametrize("fconv", ["rusanov", "roe"])
@pytest.mark.parametrize("order", [1, 2, 3, 4, 5])
def test_vjp_dot_product(order, fconv, bounds):
    """The difference quotient's error is eps^2 times a third derivative plus
    1e-16 / eps of cancellation, except at the points within eps of a kink of
    the fluxes (|Vn| and the largest wave speed), a share of order eps whose
    slope is off by a factor of order one: 1e-4 covers ten of them."""
    if bounds == "periodic":
        mesh = meshgen.jitter_interior(meshgen.box_quads(5, 4, 0.0, 1.0, 0.0, 1.0), 0.02, 3)
        names = {"PERIODIC": "periodic"}
    else:
        mesh = meshgen.cylinder_omesh(4, 7, r1=3.0)
        names = {"WALL": "wall_ns_adi", "FARFIELD": "char"}
    p = make_params(order, True, gamma=1.4, prandtl=0.71, mu=1e-2, ldg_b=0.5, ldg_tau=0.1, fconv=fconv,
                    V_fs=(0.3, 0.1, 0.0))
    s = FRSolver(mesh, p, names)
    rng = np.random.default_rng(order)
    X = s.plan.get("coord_spts").reshape(s.nspts, 2, s.neles)
    U = np.empty(s.state_shape)
    U[:, 0] = 1.0 + 0.1 * np.sin(3 * X[:, 0] + X[:, 1])
    U[:, 1] = 0.3 + 0.1 * np.cos(2 * X[:, 1])
    U[:, 2] = 0.1 + 0.1 * np.sin(2 * X[:, 0])
    U[:, 3] = 2.6 + 0.1 * np.cos(X[:, 0] - X[:, 1])
    lam, v = rng.standard_normal(s.state_shape), rng.standard_normal(s.state_shape)
    eps = 1e-6
    dR = (s.residual(U + eps * v) - s.residual(U - eps * v)) / (2 * eps)
    s.set_state(U)
    bar = s.vjp(lam)
    assert np.array_equal(bar, s.vjp(lam))
    a, b = float((lam * dR).sum()), float((bar * v).sum())
    scale = np.linalg.norm(lam * dR)
    assert abs(a - b) <= 1e-4 * scale
