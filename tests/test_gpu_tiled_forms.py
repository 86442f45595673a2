"""The tiled kernel's ragged rows (row length no multiple of four floats) and residual epilogue, forced, at the sizes
where they can go wrong: rows split into pieces and many rows per tile, tensors that end 1 - 3 floats behind a 16-byte
boundary, blocks with a single tile, a channel per block and many, one sample.  Checked against the float64 computation
of tests/util.py; the calls whose outputs share memory with their inputs are compared with the plain kernel's."""
import numpy as np
import pytest
import torch

from tests.test_gpu_fused import dev, host, run_fused
from tests.test_gpu_random_shapes import run_add_act
from tests.util import check_layer_own_mask, make_inputs

pytestmark = pytest.mark.gpu

RAGGED = [(7, 3, 9, 13), (1, 5, 1, 163), (300, 3, 13, 13), (64, 7, 15, 15), (9, 5, 55, 55), (3, 3, 1, 8191), (2, 3, 97, 173),
          (1, 3, 1, 65543), (33, 1, 31, 33), (2, 13, 257, 65), (700, 3, 33, 31)]
ALIGNED = [(9, 6, 28, 28), (3, 2, 56, 56), (40, 24, 56, 56), (2, 3, 160, 120), (1, 2, 16, 16), (2, 150, 32, 36)]


@pytest.fixture
def tiled():
    from anode_b200 import ops
    ops.set_kernel("tiled")
    yield ops
    ops.set_kernel("auto")


@pytest.mark.parametrize("shape", RAGGED)
def test_ragged_rows(tiled, shape):
    d = make_inputs(shape, seed=sum(shape), loc=3.0, scale=2.0)
    got, ws = run_fused(tiled, d)
    check_layer_own_mask(d, got, "%r " % (shape,))
    for _ in range(3):                       # the same workspace, the next launches: bit-identical
        again, _ = run_fused(tiled, d, ws=ws)
        for k in ("y", "dx", "mean", "var"):
            assert np.array_equal(again[k], got[k]), (shape, k)


@pytest.mark.parametrize("shape", RAGGED + ALIGNED)
@pytest.mark.parametrize("slope", [0.0, 0.1])
def test_residual_epilogue(tiled, shape, slope):
    d = make_inputs(shape, seed=sum(shape), loc=0.5, scale=2.0)
    res = np.random.default_rng(5).standard_normal(shape).astype(np.float32)
    got = run_add_act(tiled, d, res, slope)
    check_layer_own_mask(d, got, "%r slope %g " % (shape, slope), residual=res, slope=slope)


@pytest.mark.parametrize("at", [0.0, 30.0, 100.0])
@pytest.mark.parametrize("shape,residual", [((64, 12, 55, 55), False), ((64, 12, 55, 55), True), ((9, 5, 31, 33), False),
                                            ((64, 8, 56, 56), False), ((64, 8, 56, 56), True), ((6, 3, 160, 121), False)])
def test_rows_that_begin_far_from_the_mean(tiled, shape, residual, at):
    """The first element of every row (the corner of the image) lies at many standard deviations.  A thread adds up at most
    16384 / 256 = 64 squares one after another, about a shift that is within two deviations of the mean, so the variance is
    off by at most 64 roundings of 2^-24 on 1 + 2^2 times its size, and typically by far less."""
    d = make_inputs(shape, seed=sum(shape), loc=0.0, scale=1.0)
    d["x"][:, :, 0, 0] = at
    x = d["x"].astype(np.float64)
    want = x.var(axis=(0, 2, 3)) + 1e-5
    got = run_add_act(tiled, d, np.zeros(shape, np.float32), 0.0) if residual else run_fused(tiled, d)[0]
    err = float(np.max(np.abs(got["var"] - want) / want))
    print("%r residual %d first element %g: relative error of the variance %.1e" % (shape, residual, at, err))
    assert err < 5 * 64 * 2.0 ** -24, err


@pytest.mark.parametrize("shape", [(7, 3, 13, 13), (64, 7, 15, 15), (700, 3, 33, 31), (40, 24, 56, 56), (2, 3, 160, 120)])
@pytest.mark.parametrize("form", ["separate", "dres is dy", "dres is y", "dres is x", "no dres", "dx is dy", "dx is x", "accumulate"])
def test_outputs_over_inputs(tiled, shape, form):
    """Every output that may take an input's place, and the accumulating write, as the plain kernel does it; a residual
    call between ordinary calls of the same layer on one workspace leaves both right."""
    outputs_over_inputs(tiled, shape, form, "tiled")


@pytest.mark.parametrize("shape", [(1841, 15, 1, 165), (2123, 21, 1, 139)])
def test_plain_and_tiled_calls_share_a_workspace(shape):
    """Ragged rows whose residual epilogue goes to the plain kernel while the ordinary calls are the tiled one's."""
    from anode_b200 import ops
    assert [ops.serving_kernel(shape, 1, residual=r) for r in (False, True)] == [("tiled" if shape[3] > 160 else "plain"), "plain"]
    outputs_over_inputs(ops, shape, "separate", "auto")


def outputs_over_inputs(ops, shape, form, kernel_name):
    d = make_inputs(shape, seed=3, loc=0.5, scale=2.0)
    y_h = np.maximum(np.random.default_rng(4).standard_normal(shape), 0).astype(np.float32)
    c = shape[1]
    mean = d["x"].mean(axis=(0, 2, 3), dtype=np.float64).astype(np.float32)
    var = (d["x"].astype(np.float64).var(axis=(0, 2, 3)) + 1e-5).astype(np.float32)
    wss = {}

    def call(kernel):
        ops.set_kernel(kernel)
        x, dy, y = dev(d["x"]), dev(d["dy"]), dev(y_h)
        dres = {"dres is dy": dy, "dres is y": y, "dres is x": x, "no dres": None}.get(form, torch.full_like(x, float("nan")))
        dx = {"dx is dy": dy, "dx is x": x}.get(form, torch.ones_like(x))
        dg, db = torch.zeros(c, device="cuda"), torch.zeros(c, device="cuda")
        ws = wss.setdefault(kernel, ops.Workspace(*ops.dims_of(x), x.device))
        ops.BatchNormalize2dAddActFusedOp.adjoint(
            [0, 1], dy, x, y, dev(mean), dev(var), dx, dres, dev(d["gamma"]), dev(d["beta"]), dg, db, 0.1,
            cap=ops.WriteCap.Accumulate if form == "accumulate" else ops.WriteCap.Assign, workspace=ws)
        assert ws.status() == 0
        return [host(t) for t in (dx, dres, dg, db) if t is not None], ws

    try:
        want, _ = call("plain")
        for _ in range(3):
            got, ws = call(kernel_name)
            for g, w in zip(got, want):
                assert np.allclose(g, w, rtol=1e-4, atol=1e-5 + 1e-4 * float(np.sqrt(np.mean(w.astype(np.float64) ** 2))))
            run, _ = run_fused(ops, d, ws=ws)
            check_layer_own_mask(d, run, "%r between residual calls " % (shape,))
    finally:
        ops.set_kernel("auto")
