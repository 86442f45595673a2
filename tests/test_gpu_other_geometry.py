"""Layers whose launch shape is chosen by an estimate: units and clusters of the streaming kernel other than its first rule's, and the
register-resident kernel with fewer registers, where that is one wave of blocks in the place of two; against float64."""
import numpy as np
import pytest

from tests.test_gpu_fused import run_fused
from tests.test_gpu_random_shapes import run_add_act
from tests.test_serving_kernel import stream_geometry
from tests.util import check_layer_own_mask, make_inputs

STREAM = [(148, 750, 1, 38), (1148, 44, 1, 80), (20, 1998, 1, 102), (285, 484, 1, 30), (3865, 36, 1, 18), (188, 356, 1, 39)]
REGISTER = [(225, 56, 1, 80), (6, 278, 1, 354), (108, 84, 1, 29), (3, 239, 1, 1451), (28, 1910, 1, 20)]


@pytest.mark.parametrize("shape", STREAM)
def test_units_clusters_and_groups_fit(shape):
    n, c, d0 = shape[0], shape[1], shape[3]
    for direction in (0, 1):
        g = stream_geometry(shape, direction)
        vectors = g["cb"] * d0 // 4
        assert g["applies"] == 1 and g["cb"] * d0 % 4 == 0 and g["cb"] <= 128 and g["cb"] * g["cluster"] <= 1024 and g["units"] == -(-c // g["cb"])
        assert g["cluster"] in (1, 2, 4, 8, 16) and g["cluster"] * g["rows"] >= n and 1 <= g["groups"] <= g["rows"]
        assert g["groups"] * vectors <= g["threads"] <= 256


@pytest.mark.gpu
@pytest.mark.parametrize("kernel,shape", [("stream", s) for s in STREAM] + [("register", s) for s in REGISTER])
def test_results(kernel, shape):
    from anode_b200 import ops
    ops.set_kernel(kernel)
    try:
        d = make_inputs(shape, seed=sum(shape), loc=2.0, scale=2.0)
        got, _ = run_fused(ops, d)
        assert ops.last_kernel() == kernel
        check_layer_own_mask(d, got, "%r " % (shape,))
        res = np.random.default_rng(5).standard_normal(shape).astype(np.float32)
        got = run_add_act(ops, d, res, 0.1)
        check_layer_own_mask(d, got, "%r residual " % (shape,), residual=res, slope=0.1)
    finally:
        ops.set_kernel("auto")
