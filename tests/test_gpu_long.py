"""The kernel for small layers of long rows, forced, at the sizes where its walk has remainders: rows of every remainder by four, a
tensor that ends inside a vector, one row and many, channels of less than a block's and of many batches, clusters of every size; its
index arithmetic on the CPU; outputs over inputs, channels with a NaN or an infinity; and where it takes another kernel's place."""
import ctypes

import numpy as np
import pytest

from tests.test_gpu_fused import run_fused
from tests.test_gpu_random_shapes import run_add_act
from tests.test_gpu_tiled_forms import outputs_over_inputs
from tests.util import check_layer_own_mask, make_inputs

SHAPES = [(1, 3, 64, 64, 8), (2, 3, 1, 38421), (1, 1, 1, 17), (3, 2, 1, 16), (1, 1, 3, 173), (7, 5, 13, 31), (41, 6, 16, 16), (1, 3, 1, 262147), (9, 40, 1, 1030),
          (2, 301, 1, 1783), (5, 77, 1, 334), (1, 700, 1, 1021), (66, 4, 1, 2050), (1, 2, 1, 40003), (33, 1, 5, 5)]


def long_geometry(shape, direction, residual):
    from anode_b200 import _lib
    d0 = int(np.prod(shape[2:]))
    out = (ctypes.c_uint32 * 7)()
    assert _lib.load().anode_gpu_batch_norm_long_geometry(d0, shape[1], shape[0], direction, residual, out) == 0
    return dict(zip(["applies", "cluster", "stride", "per_row", "total", "step_rows", "step_col"], list(out)))


@pytest.mark.parametrize("shape", [s for s in SHAPES if np.prod(s) < 2e5])
@pytest.mark.parametrize("direction,residual", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_every_element_has_one_lane(shape, direction, residual):
    n, c, d0 = shape[0], shape[1], int(np.prod(shape[2:]))
    g = long_geometry(shape, direction, residual)
    assert g["applies"] == 1 and g["cluster"] in (1, 2, 4, 8, 16) and g["stride"] == 256 * g["cluster"]
    rs, total = c * d0, n * c * d0
    seen = np.zeros(total, np.int32)
    for ch in range(c):
        for j0 in range(min(g["stride"], g["total"])):
            count = (g["total"] - j0 - 1) // g["stride"] + 1
            row = j0 // g["per_row"]
            at, col = row * rs + ch * d0, j0 - row * g["per_row"]
            for _ in range(count):                      # the kernel's place() and advance()
                mis = at % 4 if d0 % 4 else 0
                v, past = 4 * col, d0 + mis
                lo, hi = (mis if col == 0 else 0), max(0, min(4, past - v))
                if lo < hi:
                    start = at - mis + v
                    assert start % 4 == (0 if d0 % 4 else at % 4)
                    seen[start + lo:start + hi] += 1
                    assert (np.arange(start + lo, start + hi) // d0 % c == ch).all()
                at += g["step_rows"] * rs
                col += g["step_col"]
                if col >= g["per_row"]:
                    col -= g["per_row"]
                    at += rs
    assert (seen == 1).all()


@pytest.fixture
def long_rows():
    from anode_b200 import ops
    ops.set_kernel("long")
    yield ops
    ops.set_kernel("auto")


def flat(shape):
    return shape if len(shape) == 4 else shape[:3] + (shape[3] * shape[4],)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES + [(4, 260, 1, 16384)])
def test_layers(long_rows, shape):
    ops, shape = long_rows, flat(shape)
    d = make_inputs(shape, seed=sum(shape), loc=3.0, scale=2.0)
    got, ws = run_fused(ops, d)
    served = ops.serving_kernel(shape, 1)
    assert ops.last_kernel() == ("long" if served in ("tiled", "register", "plain") else served)
    check_layer_own_mask(d, got, "%r " % (shape,))
    again, _ = run_fused(ops, d, ws=ws)
    for k in ("y", "dx", "mean", "var"):
        assert np.array_equal(again[k], got[k]), (shape, k)
    res = np.random.default_rng(5).standard_normal(shape).astype(np.float32)
    for slope in (0.0, 0.1):
        got = run_add_act(ops, d, res, slope)
        check_layer_own_mask(d, got, "%r slope %g " % (shape, slope), residual=res, slope=slope)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(13, 6, 1, 3001), (13, 6, 1, 3004)])
@pytest.mark.parametrize("form", ["dres is dy", "dres is y", "dres is x", "no dres", "dx is dy", "dx is x", "accumulate"])
def test_outputs_over_inputs(shape, form):
    from anode_b200 import ops
    outputs_over_inputs(ops, shape, form, "long")


@pytest.mark.gpu
@pytest.mark.parametrize("row", [2001, 2004])
def test_a_channel_with_a_nan_or_an_infinity_leaves_its_neighbours_alone(long_rows, row):
    shape = (30, 9, 1, row)
    d = make_inputs(shape, seed=9, loc=1.0, scale=2.0)
    want, _ = run_fused(long_rows, d)
    d["x"][3, 4, 0, 0], d["x"][29, 4, 0, row - 1], d["x"][5, 6, 0, row - 1] = np.nan, np.inf, -np.inf
    got, _ = run_fused(long_rows, d)
    assert long_rows.last_kernel() == "long" and not np.isfinite(got["var"][[4, 6]]).any()
    rest = [i for i in range(9) if i not in (4, 6)]
    for k in ("y", "dx"):
        assert np.array_equal(got[k][:, rest], want[k][:, rest]), k


@pytest.mark.gpu
@pytest.mark.parametrize("shape,launched", [((64, 8, 56, 56), "long"), ((1, 4, 1, 254072), "long"), ((8, 217, 1, 2678), "long"),
                                            ((2, 3, 1, 1403220), "tiled"), ((256, 16, 56, 56), "tiled"), ((2, 512, 7, 7), "register")])
def test_where_it_is_launched(shape, launched):
    from anode_b200 import ops
    d = make_inputs(shape, seed=1, loc=1.0, scale=2.0)
    got, _ = run_fused(ops, d)
    assert ops.last_kernel() == launched
    check_layer_own_mask(d, got, "%r " % (shape,))
