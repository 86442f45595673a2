"""Which kernel serves a call, and how many launches a synchronized step takes (no GPU needed)."""
import ctypes

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


def test_forcing_the_streaming_kernel_or_its_form_for_large_layers():
    ops.set_kernel("band")
    try:
        assert [ops.serving_kernel((1024, 2048, 7, 7), d) for d in (0, 1)] == ["stream"] * 2      # (its family by shape)
        assert ops.serving_kernel((100, 1024, 14, 14), 0) == "stream"                              # where "auto" takes another one
        assert ops.serving_kernel((64, 16, 7, 7), 0) != "stream"                                   # a layer that has no band form
    finally:
        ops.set_kernel("auto")
    assert "band" not in ops.KERNELS and ops.serving_kernel((100, 1024, 14, 14), 0) == "register"


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["tiled", "cluster", "resident", "plain", "register", "stream", "band"])
def test_a_forced_kernel_is_the_one_that_was_launched(name):
    """A large layer of short rows, which the band kernel serves unless another one is forced; and the forms of other shapes."""
    shape = {"tiled": (9, 5, 55, 55), "resident": (16, 8, 56, 56), "cluster": (64, 96, 7, 7)}.get(name, (1283, 244, 7, 7))
    x = torch.randn(shape, device="cuda")
    layer = ops.FusedBatchNormRelu(shape[1])
    ops.set_kernel(name)
    try:
        layer.forward(x)
        first = ops.last_kernel()
        layer.backward(x)
        assert [first, ops.last_kernel()] == [name] * 2
    finally:
        ops.set_kernel("auto")
    if name == "stream":
        layer.forward(x)
        assert ops.last_kernel() == "band"


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


def routes(shape):
    """Kernels of the plain forward and backward and of the residual epilogue's, on one GPU."""
    return tuple(ops.serving_kernel(shape, d, residual=r) for r in (False, True) for d in (0, 1))


STREAM_FIELDS = ["applies", "cb", "units", "cluster", "rows", "groups", "threads"]


def stream_geometry(shape, direction):
    d0, c, n = ops.dims_of(torch.empty(shape, device="meta"))
    out = (ctypes.c_uint32 * 7)()
    assert _lib.load().anode_gpu_batch_norm_stream_geometry(d0, c, n, direction, out) == 0
    return dict(zip(STREAM_FIELDS, list(out)))


@pytest.mark.parametrize("shape", [(1411, 128, 7, 7), (1500, 4, 7, 9), (4099, 16, 2, 2), (1025, 512, 4, 4), (40001, 8, 1, 5),
                                   (6688, 120, 1, 11), (724, 524, 1, 11), (7663, 4, 1, 412), (333, 257, 12, 12), (3, 4, 3, 3),
                                   (1, 4, 16, 16), (5, 128, 1, 4), (2048, 2048, 7, 7), (43, 832, 1, 183), (596, 1860, 1, 9)])
def test_streaming_geometry(shape):
    """Units of 16-byte aligned runs, clusters whose blocks cover the samples, records and columns that fit the block's."""
    d0, c, n = ops.dims_of(torch.empty(shape, device="meta"))
    for direction in (0, 1):
        g = stream_geometry(shape, direction)
        assert g["applies"] == 1
        vectors = g["cb"] * d0 // 4
        assert g["cb"] * d0 % 4 == 0 and g["cb"] <= 128 and g["cb"] * g["cluster"] <= 1024
        assert g["units"] == -(-c // g["cb"])
        assert g["cluster"] in (1, 2, 4, 8, 16) and g["cluster"] * g["rows"] >= n and g["rows"] <= n
        assert 1 <= g["groups"] <= g["rows"] and g["groups"] * vectors <= g["threads"] <= 256
    assert stream_geometry((9, 4, 1, 3), 0)["applies"] == 0            # rows of less than four floats
    assert stream_geometry((9, 3, 1, 7), 0)["applies"] == 0            # no aligned run


@pytest.mark.parametrize("shape,blocks", [((6688, 120, 1, 11), 160), ((3067, 108, 1, 22), 288), ((724, 524, 1, 11), 300), ((5879, 15, 1, 76), 100)])
def test_layers_of_few_channels_are_split_into_enough_units(shape, blocks):
    for direction in (0, 1):
        g = stream_geometry(shape, direction)
        assert g["units"] * g["cluster"] >= blocks, g


@pytest.mark.parametrize("shape", [(43, 832, 1, 183), (230, 568, 1, 46), (454, 304, 1, 35), (995, 1892, 1, 6)])
def test_small_layers_take_one_wave_of_blocks(shape):
    g = stream_geometry(shape, 0)
    assert g["units"] * g["cluster"] <= 3 * 148 * 8 // 7, g


def test_routes_of_layers_that_the_streaming_kernel_leaves_to_others():
    # few channels, hundreds of samples a thread: the tiled kernel where it can, for odd rows the plain one in one pass
    assert routes((7663, 4, 1, 412)) == ("tiled",) * 4
    assert routes((5111, 9, 1, 420)) == ("tiled",) * 4
    assert routes((4976, 11, 1, 260)) == ("stream",) * 4
    assert routes((17770, 12, 1, 27)) == ("stream", "stream", "plain", "stream")
    assert routes((18431, 12, 1, 37)) == ("stream",) * 4
    assert routes((57124, 7, 1, 32)) == ("stream",) * 4


def test_routes_of_scalar_rows_between_the_register_resident_kernel_and_the_others():
    reg = "register"
    # teams of more than one wave of blocks: backward passes and the residual epilogue go to the streaming kernel
    assert routes((103, 304, 1, 53)) == (reg, "stream", "stream", "stream")
    assert routes((115, 704, 1, 29)) == (reg, "stream", "stream", "stream")
    # one wave, few samples, or clusters of sixteen there: they stay
    assert routes((19, 728, 1, 145)) == (reg,) * 4
    assert routes((15, 1516, 1, 130)) == (reg,) * 4
    assert routes((336, 212, 1, 29)) == (reg,) * 4
    # rows of 1 - 3 floats: the shared-memory kernel where its blocks are resident at once
    assert routes((1024, 512, 1, 3))[0] == reg and routes((1024, 512, 1, 3))[2] == "cluster"
    assert routes((256, 1000, 1, 1)) == (reg,) * 4
    # rows without an aligned run: the residual epilogue's backward pass goes to the tiled kernel earlier
    assert routes((26, 551, 1, 431)) == (reg, reg, reg, "tiled")
    # small layers
    for shape in ((2, 512, 7, 7), (32, 64, 28, 28), (1, 53, 39, 25), (1, 260, 128, 128)):
        assert routes(shape) == (reg,) * 4


def test_routes_of_the_residual_epilogue_on_long_rows():
    for shape in ((256, 256, 56, 56), (331, 19, 1, 4392), (126, 16, 1, 3776), (256, 64, 56, 56)):
        assert routes(shape)[2:] == ("tiled", "tiled"), shape
    # ragged rows below which the plain kernel is the faster form
    assert routes((2123, 21, 1, 139))[2:] == ("plain", "plain")
    assert routes((1841, 15, 1, 165)) == ("tiled", "tiled", "tiled", "plain")
    assert routes((966, 13, 1, 191)) == ("tiled",) * 4


def test_ragged_tiles_hold_equally_many_rows():
    lib = _lib.load()
    for d0, c, n in ((131, 106, 846), (135, 210, 371), (3025, 95, 64), (1001, 7, 50)):
        for direction in (0, 1):
            out = (ctypes.c_uint32 * 12)()
            assert lib.anode_gpu_batch_norm_tiled_geometry(d0, c, n, direction, out) == 0
            if out[0] and out[2] >= d0:
                tiles = -(-n // out[1])
                assert out[3] == tiles and n - (tiles - 1) * out[1] > out[1] - tiles, (d0, c, n, list(out))


@pytest.mark.parametrize("shape,one,residual", [
    # medium rows: the tiled kernel takes the large layers, backward passes and the residual epilogue earlier
    ((256, 256, 20, 20), ("tiled", "tiled"), ("tiled", "tiled")), ((128, 512, 28, 28), ("tiled", "tiled"), ("tiled", "tiled")),
    ((256, 256, 24, 24), ("tiled", "tiled"), ("tiled", "tiled")),
    ((140, 128, 28, 28), ("tiled", "tiled"), ("tiled", "tiled")), ((100, 300, 24, 24), ("register", "tiled"), ("tiled", "tiled")),
    # not the ordinary layers, nor rows of less than 320 floats beyond the forward pass
    ((279, 32, 28, 28), ("tiled", "tiled"), ("stream", "stream")), ((4096, 64, 16, 16), ("tiled", "stream"), ("stream", "stream")),
    ((549, 32, 16, 16), ("stream", "stream"), ("stream", "stream")),
    # channels that a team holds: backward passes and the residual epilogue, where a channel is more than a tile or two
    ((16, 512, 56, 56), ("register", "tiled"), ("tiled", "tiled")), ((1, 2048, 100, 100), ("register", "register"), ("register", "register")),
    ((25, 1024, 28, 28), ("register", "register"), ("register", "register"))])
def test_routes_between_the_streaming_the_register_resident_and_the_tiled_kernel(shape, one, residual):
    assert routes(shape) == one + residual


@pytest.mark.parametrize("shape,kernel", [((96, 1024, 18, 18), "register"), ((98, 1024, 16, 20), "register"), ((78, 1024, 20, 20), "register"),
                                          ((65, 1024, 22, 22), "tiled"), ((47, 1024, 26, 26), "tiled")])
def test_channels_that_a_team_holds_stay_there_below_rows_of_480_floats(shape, kernel):
    assert routes(shape) == ("register", kernel, kernel, kernel)
