"""The streaming cluster kernel, forced, at the sizes where its splits have remainders: units of fewer channels at the end,
columns shared by two channels, blocks with few or no samples, one batch and many, one sample and one group, the smallest
and largest run and the most channels of a unit; checked against the float64 computation of tests/util.py, the calls whose
outputs lie over inputs against the plain kernel.  Every call is asserted to be served by this kernel."""
import numpy as np
import pytest

from tests.test_gpu_fused import run_fused
from tests.test_gpu_random_shapes import run_add_act
from tests.test_gpu_tiled_forms import outputs_over_inputs
from tests.util import check_layer_own_mask, make_inputs

pytestmark = pytest.mark.gpu

SHAPES = [(1411, 128, 7, 7), (1500, 4, 7, 9), (4099, 16, 2, 2), (1025, 512, 4, 4), (700, 60, 14, 14), (2000, 20, 11, 11),
          (40001, 8, 1, 5), (3001, 6, 5, 6), (600, 36, 15, 17), (9000, 4, 3, 3), (333, 257, 12, 12),
          (65, 8, 1, 516),            # clusters of sixteen, three of them without a sample
          (5, 128, 1, 4), (7, 130, 2, 2), (3, 4, 3, 3), (1, 4, 16, 16), (33, 1, 1, 4), (2, 3, 1, 1024),
          (6688, 20, 1, 11), (1999, 12, 1, 412), (43, 832, 1, 183)]


@pytest.fixture
def stream():
    from anode_b200 import ops
    ops.set_kernel("stream")
    yield ops
    ops.set_kernel("auto")


@pytest.mark.parametrize("shape", SHAPES)
def test_layers_of_short_rows(stream, shape):
    ops = stream
    assert [ops.serving_kernel(shape, d) for d in (0, 1)] == ["stream"] * 2
    d = make_inputs(shape, seed=sum(shape), loc=3.0, scale=2.0)
    got, ws = run_fused(ops, d)
    check_layer_own_mask(d, got, "%r " % (shape,))
    again, _ = run_fused(ops, d, ws=ws)
    for k in ("y", "dx", "mean", "var"):
        assert np.array_equal(again[k], got[k]), (shape, k)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("slope", [0.0, 0.1])
def test_residual_epilogue(stream, shape, slope):
    ops = stream
    assert [ops.serving_kernel(shape, d, residual=True) for d in (0, 1)] == ["stream"] * 2
    d = make_inputs(shape, seed=sum(shape), loc=0.5, scale=2.0)
    res = np.random.default_rng(5).standard_normal(shape).astype(np.float32)
    got = run_add_act(ops, d, res, slope)
    check_layer_own_mask(d, got, "%r slope %g " % (shape, slope), residual=res, slope=slope)


@pytest.mark.parametrize("form", ["dres is dy", "dres is y", "dres is x", "no dres", "dx is dy", "dx is x", "accumulate"])
def test_outputs_over_inputs(form):
    from anode_b200 import ops
    outputs_over_inputs(ops, (1411, 12, 7, 7), form, "stream")
