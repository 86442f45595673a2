"""The band kernel's geometry (no GPU needed): bands, boxes and slots that the tensor copies can take, tiles that stay in tensor
memory, units whose words a warp can merge, and the layers that are handed to it."""
import ctypes

import pytest
import torch

from anode_b200 import _lib, ops

FIELDS = ["taken", "cb", "units", "groups", "vpt", "rows", "tiles", "grid", "look", "boxes", "box4", "box_bytes", "slots", "stride", "smem", "shift"]
SHAPES = [(1024, 2048, 7, 7), (256, 1024, 14, 14), (128, 2048, 7, 7), (1283, 244, 7, 7), (300, 257, 14, 14), (500, 2003, 4, 4), (2000, 64, 11, 11),
          (80, 900, 15, 15), (1000, 2602, 2, 3), (60, 1004, 16, 17), (4096, 64, 16, 16), (801, 5002, 2, 2), (700, 4500, 1, 5), (1, 1004, 17, 18)]
# more words to a unit than a warp merges, or units that fit no thread; rows of three floats; channels whose bands are no whole vectors
REFUSED = [(2500, 1000, 2, 2), (4099, 2048, 1, 5), (8000, 20, 11, 11), (9000, 2000, 1, 3), (2000, 1001, 1, 7)]


def band(shape, direction, residual):
    out = (ctypes.c_uint32 * 16)()
    assert _lib.load().anode_gpu_batch_norm_band_geometry(*ops.dims_of(torch.empty(shape, device="meta")), direction, residual, out) == 0
    return dict(zip(FIELDS, out))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("direction", [0, 1])
@pytest.mark.parametrize("residual", [0, 1])
def test_geometry(shape, direction, residual):
    d0, c, n = ops.dims_of(torch.empty(shape, device="meta"))
    g = band(shape, direction, residual)
    assert g["cb"] > 0
    vectors, kept, planes = g["cb"] * d0 // 4, 1 + direction, 1 + direction + (direction and residual)
    assert g["cb"] * d0 % 4 == 0 and g["cb"] <= min(c, 32) and g["units"] == -(-c // g["cb"])
    # a thread per column and group; the tile's rows cover the samples, the last tile is not empty
    assert g["groups"] * vectors <= 256 and g["rows"] == g["groups"] * g["vpt"] and (g["tiles"] - 1) * g["rows"] < n <= g["tiles"] * g["rows"]
    # tensor copies: boxes of at most 256 x 256, rows of 16-byte multiples, places of 128-byte multiples
    assert g["boxes"] * g["box4"] >= vectors > (g["boxes"] - 1) * g["box4"] and g["box4"] <= 64 and g["rows"] <= 256
    assert g["box_bytes"] % 128 == 0 and g["box_bytes"] >= g["rows"] * g["box4"] * 16
    assert g["boxes"] * planes <= 32 and g["stride"] == planes * g["boxes"] * g["box_bytes"]
    assert 2 <= g["slots"] <= 8 and g["smem"] <= 227 * 1024
    # tiles in tensor memory: 512 columns of which four warps of eight share a lane, four columns a vector
    assert kept * g["vpt"] * 4 * (g["look"] + 1) <= 256
    # a unit is reduced before it is applied, and its words fit what a warp merges
    assert g["look"] * g["grid"] >= g["tiles"] + g["grid"] and g["tiles"] * g["cb"] <= 512
    assert (32 >> g["shift"]) >= g["cb"] and 4 * g["rows"] * c * d0 < 1 << 32


@pytest.mark.parametrize("shape", REFUSED)
def test_shapes_that_the_kernel_cannot_take(shape):
    for direction in (0, 1):
        for residual in (0, 1):
            assert not any(band(shape, direction, residual).values())


def test_layers_that_are_handed_over():
    def taken(shape):
        return tuple(band(shape, d, r)["taken"] for r in (0, 1) for d in (0, 1))
    assert taken((1024, 2048, 7, 7)) == (1, 1, 1, 1)
    assert taken((128, 2048, 7, 7)) == (0, 1, 1, 1)              # forward passes of 13 M elements are not
    assert taken((32, 2048, 7, 7)) == (0, 0, 0, 0)
    assert taken((8000, 20, 11, 11)) == (0, 0, 0, 0)             # more words to a unit than a warp merges in time
    assert taken((256, 512, 20, 20)) == (0, 0, 0, 0)             # rows that the tiled kernel takes
    # forward passes that the streaming kernel has in one wave of resident blocks stay with it longer
    assert taken((320, 400, 11, 11)) == (0, 1, 1, 1) and taken((200, 2048, 7, 7)) == (0, 1, 1, 1) and taken((224, 2048, 7, 7)) == (1, 1, 1, 1)
    assert taken((112, 2048, 7, 7)) == (0, 1, 0, 1) and taken((512, 2048, 4, 4)) == (1, 1, 1, 1) and taken((548, 596, 1, 46)) == (1, 1, 1, 1)
    # channels that a team's registers hold, where the band kernel is the faster one
    assert tuple(ops.serving_kernel((256, 1024, 14, 14), d, residual=r) for r in (False, True) for d in (0, 1)) == ("stream",) * 4
    assert tuple(ops.serving_kernel((100, 1024, 14, 14), d, residual=r) for r in (False, True) for d in (0, 1)) == ("register", "stream", "stream", "stream")
    assert tuple(ops.serving_kernel((64, 1024, 14, 14), d, residual=r) for r in (False, True) for d in (0, 1)) == ("register",) * 4


def test_its_words_have_their_own_place_in_the_workspace():
    """A call of a shape that is handed over asks for room for two buffers of words per direction and form, behind what the others use."""
    lib = _lib.load()
    for shape in ((1024, 2048, 7, 7), (256, 1024, 14, 14)):
        words = sum(16 * g["units"] * g["tiles"] * g["cb"] for g in (band(shape, d, r) for d in (0, 1) for r in (0, 1)))
        plan = (ctypes.c_uint32 * 15)()
        d = ops.dims_of(torch.empty(shape, device="meta"))
        assert lib.anode_gpu_batch_norm_fused_plan(*d, 1, 0, 0, 0, plan, 15) == 0
        assert lib.anode_gpu_batch_norm_fused_workspace_bytes(*d) >= 2 * (plan[13] + words)


def test_the_words_of_both_directions_share_their_place():
    """A part of the workspace serves one direction: behind what the other kernels use there is room for the larger direction's words, twice
    a pair of doubles per tile and channel in each of its two forms, and no more."""
    lib = _lib.load()
    for shape in ((1024, 2048, 7, 7), (256, 2048, 7, 7), (1283, 244, 7, 7), (128, 2048, 7, 7)):      # (no other kernel keeps words of its own here)
        forms = [[band(shape, d, r) for r in (0, 1)] for d in (0, 1)]
        room = max(sum(-(-32 * g["units"] * g["tiles"] * g["cb"] // 256) * 256 for g in f if g["taken"]) for f in forms)
        d = ops.dims_of(torch.empty(shape, device="meta"))
        part = lib.anode_gpu_batch_norm_fused_workspace_bytes(*d) // 2
        plan = (ctypes.c_uint32 * 15)()
        assert lib.anode_gpu_batch_norm_fused_plan(*d, 1, 0, 0, 0, plan, 15) == 0
        assert part == plan[13] + room, (shape, plan[13], room, part)
