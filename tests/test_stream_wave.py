"""Layers whose first choice of unit and cluster makes one wave of blocks and less than a third of another: the streaming kernel
takes another unit and cluster there.  Its geometry, and its results where the last unit is narrower, the samples do not divide
by the blocks of a cluster, or one row of a unit takes a whole block; and the small layers of
scalar rows that come to it from the register-resident kernel."""
import numpy as np
import pytest

from tests.test_gpu_fused import run_fused
from tests.test_gpu_random_shapes import run_add_act
from tests.test_serving_kernel import routes, stream_geometry
from tests.util import check_layer_own_mask, make_inputs

SHAPES = [(33, 2048, 7, 7), (64, 2000, 5, 5), (35, 2044, 7, 7), (302, 233, 10, 10), (36, 482, 14, 14), (313, 911, 4, 4)]
WAVE = 3 * 148                          # blocks of 256 threads that the device holds


@pytest.mark.parametrize("shape", SHAPES)
def test_one_wave_of_blocks(shape):
    n, c, d0 = shape[0], shape[1], shape[2] * shape[3]
    g = stream_geometry(shape, 0)
    assert g["applies"] == 1 and g["units"] * g["cluster"] <= WAVE, g
    assert g["cb"] * d0 % 4 == 0 and g["cb"] <= 128 and g["cb"] * g["cluster"] <= 1024 and g["units"] == -(-c // g["cb"])
    assert g["cluster"] in (1, 2, 4, 8) and g["cluster"] * g["rows"] >= n >= g["rows"] >= g["groups"] >= 1
    assert 192 < g["groups"] * g["cb"] * d0 // 4 <= g["threads"] <= 256


@pytest.mark.parametrize("shape", [(103, 1000, 7, 7), (117, 1000, 7, 7), (365, 1000, 5, 5), (1015, 512, 4, 4), (723, 2048, 4, 4), (302, 233, 10, 10),
                                   (140, 940, 7, 7), (64, 2048, 7, 7)])
def test_no_wave_of_clusters_that_are_not_all_resident(shape):
    """Clusters of eight fill 85 per cent of the device's places, of four 94: a grid that is chosen to be one wave fits those."""
    for direction in (0, 1):
        g = stream_geometry(shape, direction)
        blocks = g["units"] * g["cluster"]
        assert blocks > WAVE or blocks <= {8: 377, 4: 416}.get(g["cluster"], WAVE), (direction, g)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES + [(103, 1000, 7, 7), (153, 940, 7, 7)])
def test_results(shape):
    from anode_b200 import ops
    ops.set_kernel("stream")
    try:
        assert [ops.serving_kernel(shape, d, residual=r) for r in (False, True) for d in (0, 1)] == ["stream"] * 4
        d = make_inputs(shape, seed=sum(shape), loc=3.0, scale=2.0)
        got, _ = run_fused(ops, d)
        check_layer_own_mask(d, got, "%r " % (shape,))
        res = np.random.default_rng(5).standard_normal(shape).astype(np.float32)
        got = run_add_act(ops, d, res, 0.1)
        check_layer_own_mask(d, got, "%r residual " % (shape,), residual=res, slope=0.1)
    finally:
        ops.set_kernel("auto")


# Rows of one float at a time in the register-resident kernel, 1 - 3 M elements: (shape, routes of routes())
LINES = [((25, 932, 1, 45), ("register",) * 3 + ("stream",)),         # one wave of teams: the residual backward alone
         ((20, 848, 1, 43), ("register",) * 4),                       # below a million elements
         ((19, 1496, 1, 57), ("register",) * 4),                      # fewer than twenty samples
         ((29, 1248, 1, 57), ("register", "stream", "stream", "stream")),
         ((25, 932, 1, 130), ("register", "register", "register", "stream")),     # two waves of the streaming kernel's blocks
         ((30, 520, 1, 145), ("register", "stream", "stream", "stream")),
         ((25, 3720, 1, 11), ("register",) * 4), ((24, 10100, 1, 11), ("register",) * 4),      # units of 92 channels
         ((29, 5156, 1, 19), ("register",) * 3 + ("stream",)), ((24, 10828, 1, 6), ("register",) + ("stream",) * 3),
         ((300, 188, 1, 23), ("register",) * 3 + ("stream",))]


@pytest.mark.parametrize("shape,want", LINES)
def test_small_layers_of_scalar_rows(shape, want):
    assert routes(shape) == want


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [s for s, w in LINES if "stream" in w])
def test_results_of_small_layers_of_scalar_rows(shape):
    from anode_b200 import ops
    d = make_inputs(shape, seed=sum(shape), loc=1.0, scale=2.0)
    got, _ = run_fused(ops, d)
    check_layer_own_mask(d, got, "%r " % (shape,))
    res = np.random.default_rng(7).standard_normal(shape).astype(np.float32)
    got = run_add_act(ops, d, res, 0.0)
    check_layer_own_mask(d, got, "%r residual " % (shape,), residual=res, slope=0.0)
