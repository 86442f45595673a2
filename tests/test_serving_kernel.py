"""Which kernel serves a call, and how many launches a synchronized step takes (no GPU needed)."""
import pytest
import torch

from anode_b200 import _lib, ops

# shape; forward and backward: on one GPU, on two ranks, both with the residual epilogue, tensors off the 16-byte boundary
ROUTES = [
    ((2, 512, 7, 7), ("register", "register"), ("cluster", "cluster"), ("register", "register"), ("cluster", "cluster"), ("register", "register")),
    ((1, 260, 128, 128), ("register", "register"), ("tiled", "tiled"), ("register", "register"), ("resident", "resident"), ("register", "register")),
    ((8, 32, 56, 56), ("register", "register"), ("tiled", "tiled"), ("register", "register"), ("resident", "resident"), ("register", "register")),
    ((64, 8, 56, 56), ("tiled", "tiled"), ("tiled", "tiled"), ("tiled", "tiled"), ("resident", "resident"), ("plain", "plain")),
    ((2048, 256, 56, 56), ("tiled", "tiled"), ("tiled", "tiled"), ("tiled", "tiled"), ("resident", "resident"), ("plain", "plain")),
    ((64, 95, 55, 55), ("tiled", "tiled"), (None, None), ("tiled", "tiled"), (None, None), ("plain", "plain")),
    ((1024, 2048, 7, 7), ("stream", "stream"), ("cluster", "cluster"), ("stream", "stream"), ("cluster", None), ("register", "register")),
    ((5, 3, 7, 7), ("register", "register"), (None, None), ("register", "register"), (None, None), ("register", "register")),
    ((512, 64, 19, 19), ("plain", "plain"), (None, None), ("plain", "plain"), (None, None), ("plain", "plain")),
]


@pytest.mark.parametrize("shape,one,two,res_one,res_two,unaligned", ROUTES)
def test_the_query_names_the_kernel_of_every_form_of_call(shape, one, two, res_one, res_two, unaligned):
    assert tuple(ops.serving_kernel(shape, d) for d in (0, 1)) == one
    assert tuple(ops.serving_kernel(shape, d, world=2) for d in (0, 1)) == two
    assert tuple(ops.serving_kernel(shape, d, residual=True) for d in (0, 1)) == res_one
    assert tuple(ops.serving_kernel(shape, d, residual=True, world=2) for d in (0, 1)) == res_two
    assert tuple(ops.serving_kernel(shape, d, aligned=False) for d in (0, 1)) == unaligned


def test_the_family_of_a_shape():
    """kernel_kind knows four kernels: those of the shapes that the register-resident and streaming kernels take over, too."""
    kind = _lib.load().anode_gpu_batch_norm_fused_kernel_kind
    for shape, family in (((1, 260, 128, 128), 1), ((16, 8, 56, 56), 1), ((64, 8, 56, 56), 1), ((32, 64, 28, 28), 2),
                          ((1024, 2048, 7, 7), 2), ((5, 3, 7, 7), 4), ((64, 95, 55, 55), 4)):
        d0, c, n = ops.dims_of(torch.empty(shape, device="meta"))
        assert [kind(d0, c, n, d) for d in (0, 1)] == [family] * 2, shape


@pytest.mark.parametrize("name", sorted(ops.KERNELS))
def test_a_forced_kernel_is_the_one_that_serves(name):
    shape = {"tiled": (9, 5, 55, 55), "cluster": (64, 96, 7, 7), "resident": (16, 8, 56, 56), "plain": (64, 8, 56, 56),
             "register": (64, 16, 14, 14), "stream": (64, 16, 7, 7), "auto": (64, 8, 56, 56)}[name]
    ops.set_kernel(name)
    try:
        assert [ops.serving_kernel(shape, d) for d in (0, 1)] == ["tiled" if name == "auto" else name] * 2
    finally:
        ops.set_kernel("auto")


class Comm:
    """Ranks of a synchronized layer, as far as it is asked for the launches of a step."""
    def __init__(self, world, exchange):
        self.world, self._exchange = world, exchange


@pytest.mark.parametrize("shape,launches", [((16, 8, 56, 56), 2), ((32, 64, 56, 56), 2), ((1, 260, 128, 128), 2), ((32, 64, 7, 7), 2),
                                            ((2, 512, 7, 7), 2), ((1024, 2048, 7, 7), 2), ((6, 3, 5, 5), 6), ((64, 95, 55, 55), 6)])
def test_launches_of_a_synchronized_step(shape, launches):
    layer = ops.SyncBatchNormRelu(shape[1], comm=Comm(2, object()), device="cpu")
    layer._x = torch.empty(shape, device="meta")            # what a forward leaves behind
    assert layer.launches_per_step == launches
    layer.comm = Comm(2, None)                              # records over NCCL: three kernels per direction
    assert layer.launches_per_step == 6
    layer.comm = Comm(1, None)
    assert layer.launches_per_step == 2
