"""The register-resident kernel, forced: teams of one warp, one block and 2, 4 and 8 blocks, channels that fill a team to the
last element and one more or less, rows of 1 - 3 floats, 4-byte and 16-byte loads, tensors off the 16-byte boundary; checked
against the float64 computation of tests/util.py, the calls whose outputs lie over inputs against the plain kernel."""
import numpy as np
import pytest
import torch

from tests.test_gpu_fused import host, run_fused
from tests.test_gpu_random_shapes import run_add_act
from tests.test_gpu_tiled_forms import outputs_over_inputs
from tests.util import check_layer_own_mask, make_inputs

pytestmark = pytest.mark.gpu

# elements of a channel: 32 lanes, 512 threads, 2, 4 and 8 blocks of 512 with 4, 8, 16 (and, forward, 32) floats a thread
SHAPES = [(1, 3, 1, 128), (1, 3, 1, 129), (1, 5, 1, 127), (128, 6, 1, 1), (129, 3, 1, 1), (43, 9, 1, 3), (64, 7, 1, 2),
          (4, 3, 1, 512), (1, 3, 1, 2049), (683, 2, 1, 3), (2, 3, 64, 64), (1, 2, 1, 8193), (17, 3, 31, 31), (4, 2, 64, 64),
          (1, 2, 1, 16385), (5, 3, 57, 57), (1, 2, 128, 256), (1, 2, 1, 32769), (1, 1, 1, 65535), (1, 1, 256, 256), (2, 1, 181, 181)]


@pytest.fixture
def register():
    from anode_b200 import ops
    ops.set_kernel("register")
    yield ops
    ops.set_kernel("auto")


@pytest.mark.parametrize("shape", SHAPES)
def test_teams(register, shape):
    assert [register.serving_kernel(shape, d) for d in (0, 1)] == ["register"] * 2
    d = make_inputs(shape, seed=sum(shape), loc=3.0, scale=2.0)
    got, ws = run_fused(register, d)
    check_layer_own_mask(d, got, "%r " % (shape,))
    again, _ = run_fused(register, d, ws=ws)
    for k in ("y", "dx", "mean", "var"):
        assert np.array_equal(again[k], got[k]), (shape, k)


@pytest.mark.parametrize("shape", [(1, 1, 1, 131071), (1, 1, 256, 512), (5, 1, 1, 26213)])
def test_largest_forward_teams(register, shape):
    """Twice as many floats a thread as the backward pass and the residual epilogue have."""
    assert register.serving_kernel(shape, 0) == "register" and register.serving_kernel(shape, 1) != "register"
    d = make_inputs(shape, seed=sum(shape), loc=3.0, scale=2.0)
    got, _ = run_fused(register, d)
    check_layer_own_mask(d, got, "%r " % (shape,))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("slope", [0.0, 0.1])
def test_residual_epilogue(register, shape, slope):
    assert [register.serving_kernel(shape, d, residual=True) for d in (0, 1)] == ["register"] * 2
    d = make_inputs(shape, seed=sum(shape), loc=0.5, scale=2.0)
    res = np.random.default_rng(5).standard_normal(shape).astype(np.float32)
    got = run_add_act(register, d, res, slope)
    check_layer_own_mask(d, got, "%r slope %g " % (shape, slope), residual=res, slope=slope)


@pytest.mark.parametrize("shape", [(9, 5, 7, 7), (4, 6, 56, 56)])
@pytest.mark.parametrize("form", ["separate", "dres is dy", "dres is y", "dres is x", "no dres", "dx is dy", "dx is x", "accumulate"])
def test_outputs_over_inputs(register, shape, form):
    outputs_over_inputs(register, shape, form, "register")


@pytest.mark.parametrize("shape", [(2, 64, 7, 7), (4, 6, 56, 56), (3, 5, 16, 16)])
def test_tensors_off_the_16_byte_boundary(register, shape):
    """The same numbers from tensors that start 4 bytes further: the 4-byte form of the kernel."""
    d = make_inputs(shape, seed=1, loc=0.5, scale=2.0)
    num, c = d["x"].size, shape[1]

    def placed(a):
        t = torch.full((num + 1,), float("nan"), device="cuda")[1:].view(shape)
        return t if a is None else t.copy_(torch.from_numpy(a))
    x, dy, y, dx = placed(d["x"]), placed(d["dy"]), placed(None), placed(None)
    assert x.data_ptr() % 16 == 4
    assert [register.serving_kernel(shape, k, aligned=False) for k in (0, 1)] == ["register"] * 2
    v = {k: torch.zeros(c, device="cuda") for k in ("mean", "var", "run_mean", "run_var", "dgamma", "dbeta")}
    g, b = torch.from_numpy(d["gamma"]).cuda(), torch.from_numpy(d["beta"]).cuda()
    ws = register.Workspace(*register.dims_of(x), x.device)
    register.BatchNormalize2dFusedOp.apply([0, 1], 1e-5, 0.1, x, y, v["mean"], v["var"], v["run_mean"], v["run_var"], g, b, workspace=ws)
    register.BatchNormalize2dBwdFusedOp.apply([0, 1], dy, x, v["mean"], v["var"], dx, g, b, v["dgamma"], v["dbeta"], workspace=ws)
    assert ws.status() == 0
    check_layer_own_mask(d, dict({k: host(t) for k, t in v.items()}, y=host(y), dx=host(dx)), "%r unaligned " % (shape,))
