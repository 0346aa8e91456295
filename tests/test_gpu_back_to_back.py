"""Passes queued back to back on one stream, two states in turn, every output in
a buffer of its own, against each state's first pass run alone: the same bits.
Kernels that hand traces, viscous normal fluxes, volume residuals or block sums
to the next one would show a missing dependency here as a rare difference."""
import pytest

torch = pytest.importorskip("torch")

from zefr_b200 import meshgen  # noqa: E402
from zefr_b200.solver import FRSolver, make_params  # noqa: E402

pytestmark = pytest.mark.gpu

REPEATS = 400

# name: mesh, order, viscous, flux, beta, precision, boundaries
PER = {"PERIODIC": "periodic"}
CASES = {
    "quad_euler": (lambda: meshgen.box_quads(32, 32), 3, False, "rusanov", 0.5, "fp64", PER),
    "quad_euler_mixed": (lambda: meshgen.box_quads(31, 33), 4, False, "roe", 0.5, "mixed", PER),
    "cylinder_ns": (lambda: meshgen.cylinder_omesh(24, 48), 3, True, "rusanov", 0.5, "fp64",
                    {"WALL": "wall_ns_adi", "FARFIELD": "char"}),
    "quad_ns_mixed": (lambda: meshgen.box_quads(41, 37), 4, True, "roe", 0.3, "mixed", PER),
    "tri_euler": (lambda: meshgen.box_tris(40), 1, False, "rusanov", 0.5, "fp64", PER),
    "tri_ns": (lambda: meshgen.box_tris(48), 3, True, "rusanov", 0.5, "fp64", PER),
    "tri_ns_mixed": (lambda: meshgen.box_tris(60), 4, True, "roe", -0.5, "mixed", PER),
    "hex_euler": (lambda: meshgen.box_hexes(11, 10, 9), 2, False, "rusanov", 0.5, "fp64", PER),
    "hex_ns": (lambda: meshgen.box_hexes(10, 9, 11), 3, True, "roe", 0.5, "fp64", PER),
    "hex_ns_traces": (lambda: meshgen.box_hexes(9, 9, 8), 2, True, "rusanov", 0.3, "fp64", PER),
    "hex_ns_mixed": (lambda: meshgen.box_hexes(12, 11, 10), 3, True, "roe", 0.5, "mixed", PER),
}


def _solver(name):
    mesh, order, viscous, flux, beta, precision, bounds = CASES[name]
    p = make_params(order, viscous, gamma=1.4, prandtl=0.71, mu=2e-3, ldg_b=beta, ldg_tau=0.1, fconv=flux,
                    precision=precision, dt=1e-5, V_fs=(0.2, 0.0, 0.0))
    s = FRSolver(mesh(), p, bounds)
    s.set_stream(torch.cuda.current_stream().cuda_stream)
    return s


def _states(s):
    g = torch.Generator(device="cuda").manual_seed(1)
    out = []
    for _ in range(2):
        U = 0.05 * torch.randn(s.state_shape, generator=g, device="cuda", dtype=torch.float64)
        U[:, 0] += 1.0
        U[:, 1] += 0.2
        U[:, -1] += 2.5
        out.append(U)
    return out


def _run(one_pass, states, shape):
    """Bits of REPEATS queued passes against each state's pass run alone."""
    alone = []
    for U in states:
        o = torch.empty(shape, device="cuda", dtype=torch.float64)
        torch.cuda.synchronize()
        one_pass(U, o)
        torch.cuda.synchronize()
        assert torch.isfinite(o).all()
        alone.append(o)
    assert not torch.equal(*alone)
    outs = [torch.empty(shape, device="cuda", dtype=torch.float64) for _ in range(REPEATS)]
    torch.cuda.synchronize()
    for i, o in enumerate(outs):
        one_pass(states[i % 2], o)
    torch.cuda.synchronize()
    bad = [i for i, o in enumerate(outs) if not torch.equal(o, alone[i % 2])]
    assert not bad, f"{len(bad)} of {REPEATS} passes differ, the first at {bad[0]}"


@pytest.mark.parametrize("op", ["step", "residual"])
@pytest.mark.parametrize("name", list(CASES))
def test_forward(name, op):
    s = _solver(name)

    def one_pass(U, out):
        s.set_state(U)
        if op == "step":
            s.step(1)
            s.get_state_device(out)
        else:
            s.compute_residual(0)
            s.get_residual_device(out, 0)

    _run(one_pass, _states(s), s.state_shape)
    s.close()


@pytest.mark.parametrize("name", ["cylinder_ns", "tri_ns", "hex_euler", "hex_ns"])
def test_adjoints(name):
    s = _solver(name)
    states = _states(s)
    lam = torch.randn(s.state_shape, generator=torch.Generator(device="cuda").manual_seed(5), device="cuda",
                      dtype=torch.float64)

    def vjp(U, out):
        s.set_state(U)
        out.copy_(s.vjp(lam))

    def step_vjp(U, out):
        out.copy_(s.rk_step_vjp(U, lam))

    _run(vjp, states, s.state_shape)
    _run(step_vjp, states, s.state_shape)
    s.close()
