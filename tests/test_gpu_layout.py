"""State import and export: every stride order, ragged tiles, both forms."""
import ctypes

import numpy as np
import pytest

from zefr_b200 import _lib, meshgen
from zefr_b200._lib import check, lib
from zefr_b200.solver import FRSolver, make_params

pytestmark = pytest.mark.gpu

_DP = ctypes.POINTER(ctypes.c_double)

# (mesh, order): one tile with padding, one thread block exactly, blocks and
# rows with remainders (25 and 6 points of 4, 8 and 125 points of 5 variables)
MESHES = [("quad", (3, 1), 2), ("quad", (16, 8), 1), ("quad", (13, 11), 4), ("tri", (9,), 2), ("hex", (3, 3, 3), 1),
          ("hex", (5, 4, 7), 4)]


def _solver(kind, n, order, precision):
    mesh = {"quad": meshgen.box_quads, "hex": meshgen.box_hexes, "tri": meshgen.box_tris}[kind](*n)
    bounds = {"PERIODIC": "periodic"}
    if kind == "quad" and 1 in n:
        bounds = {"PERIODIC": "wall_slip"}
    return FRSolver(mesh, make_params(order, precision=precision), bounds)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kind,n,order", MESHES)
@pytest.mark.parametrize("axes", [(0, 1, 2), (2, 0, 1), (2, 1, 0), (1, 0, 2)])
@pytest.mark.parametrize("pad", [0, 3])
def test_state_round_trip(kind, n, order, precision, axes, pad):
    import torch
    s = _solver(kind, n, order, precision)
    rng = np.random.default_rng(5)
    U = rng.uniform(1.0, 2.0, s.state_shape)
    # memory order `axes` of (spt, var, ele), the fastest axis padded
    shape = [s.state_shape[a] for a in axes]
    shape[-1] += pad
    view = np.zeros(shape)
    inv = np.argsort(axes)
    dense = view[..., :shape[-1] - pad].transpose(inv)
    dense[...] = U
    strides = [st // 8 for st in dense.strides]
    buf = torch.from_numpy(view).cuda()
    check(lib().zb_set_state(s.h, ctypes.cast(buf.data_ptr(), _DP), *strides, _lib.ZB_DEVICE))
    out = torch.full_like(buf, -7.0)
    torch.cuda.synchronize()
    check(lib().zb_get_state(s.h, ctypes.cast(out.data_ptr(), _DP), *strides, _lib.ZB_DEVICE))
    s.synchronize()
    got = out.cpu().numpy()
    if pad:
        assert (got[..., -pad:] == -7.0).all()
    got = got[..., :shape[-1] - pad].transpose(inv)
    if precision == "fp64":
        assert np.array_equal(got, U)
    else:
        # stored as FP32 deviations from the FP32-rounded mean: half an ulp of
        # a deviation of at most one
        assert np.abs(got - U).max() <= 2.0 ** -24
        # the mean itself: a state that is its own mean comes back exactly
        c = np.broadcast_to(np.float32([1.1, 2.2, 3.3, 4.4, 5.5])[:s.nvars].astype(np.float64)[None, :, None],
                            s.state_shape)
        s.set_state(c)
        assert np.array_equal(s.get_state(), c)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_mixed_state_without_a_finite_mean(bad):
    """A variable with no finite mean is stored as it is; the others keep theirs."""
    s = _solver("quad", (13, 11), 3, "mixed")
    U = np.random.default_rng(1).uniform(1.0, 2.0, s.state_shape)
    U[3, 2, 17] = bad
    s.set_state(U)
    got = s.get_state()
    assert np.array_equal(got[:, 2], U[:, 2].astype(np.float32).astype(np.float64), equal_nan=True)
    assert np.abs(got[:, [0, 1, 3]] - U[:, [0, 1, 3]]).max() <= 2.0 ** -24
    # the next state's mean does not see this one
    V = np.ones(s.state_shape)
    s.set_state(V)
    assert np.array_equal(s.get_state(), V)
