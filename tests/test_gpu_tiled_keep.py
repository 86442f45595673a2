"""The tiled kernel where part of a block's tiles stay in tensor memory between their two visits and the others come from L2,
in one launch: whole rows, pieces of rows, ragged rows, residual epilogue.  (The small shapes of the other tests keep all.)"""
import numpy as np
import pytest

from tests.test_gpu_fused import run_fused
from tests.test_gpu_random_shapes import run_add_act
from tests.test_tiled_keep import keep
from tests.util import check_layer_own_mask, make_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,residual", [((2048, 2, 56, 56), False), ((2043, 1, 56, 56), True), ((1500, 2, 55, 55), False),
                                            ((1501, 1, 55, 55), True), ((4, 2, 64, 128, 128), False), ((3, 2, 64, 128, 127), False)])
def test_some_tiles_stay_and_some_do_not(shape, residual):
    from anode_b200 import ops
    dims = (int(np.prod(shape[2:])), shape[1], shape[0])
    some = [0 < k["slots"] <= k["look"] for k in (keep(dims, d, int(residual), 0, 0) for d in (0, 1))]
    assert any(some), (shape, some)
    d = make_inputs(shape, seed=sum(shape), loc=0.5, scale=2.0)
    ops.set_kernel("tiled")
    try:
        if residual:
            res = np.random.default_rng(5).standard_normal(shape).astype(np.float32)
            got = run_add_act(ops, d, res, 0.1)
            check_layer_own_mask(d, got, "%r " % (shape,), residual=res, slope=0.1)
        else:
            got, ws = run_fused(ops, d)
            check_layer_own_mask(d, got, "%r " % (shape,))
            again, _ = run_fused(ops, d, ws=ws)
            for k in ("y", "dx", "mean", "var"):
                assert np.array_equal(again[k], got[k]), (shape, k)
    finally:
        ops.set_kernel("auto")


@pytest.mark.parametrize("row", [639, 640, 641, 1283])
def test_residual_rows_on_both_sides_of_the_line_below_which_tiles_stay(row):
    from anode_b200 import ops
    shape = (120, 9, 1, row)
    d = make_inputs(shape, seed=row, loc=0.5, scale=2.0)
    res = np.random.default_rng(5).standard_normal(shape).astype(np.float32)
    ops.set_kernel("tiled")
    try:
        assert bool(keep((row, 9, 120), 0, 1, 0, 0)["slots"]) == (row <= 640)
        check_layer_own_mask(d, run_add_act(ops, d, res, 0.1), "%r " % (shape,), residual=res, slope=0.1)
    finally:
        ops.set_kernel("auto")


@pytest.mark.parametrize("shape", [(120, 24, 1, 639), (120, 24, 1, 641), (64, 25, 55, 55), (3, 31, 111, 111), (1, 24, 1, 65543)])
def test_forward_rows_on_both_sides_of_the_line_below_which_tiles_stay(shape):
    from anode_b200 import ops
    d0 = shape[2] * shape[3]
    assert bool(keep((d0, shape[1], shape[0]), 0, 0, 0, 0)["slots"]) == (d0 <= 640)
    d = make_inputs(shape, seed=d0, loc=0.5, scale=2.0)
    ops.set_kernel("tiled")
    try:
        assert ops.serving_kernel(shape, 0) == "tiled"
        got, ws = run_fused(ops, d)
        check_layer_own_mask(d, got, "%r " % (shape,))
        again, _ = run_fused(ops, d, ws=ws)
        for k in ("y", "dx", "mean", "var"):
            assert np.array_equal(again[k], got[k]), (shape, k)
    finally:
        ops.set_kernel("auto")
