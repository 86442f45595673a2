"""Tiles that the tiled kernel keeps in tensor memory between their two visits: the places of the tiles that are kept at the
same time lie apart and inside a warp's columns, and every vector of a tile is dealt to one warp."""
import ctypes

import pytest

from anode_b200 import _lib

FIELDS = ["slots", "kept", "place", "dealt", "column", "before", "vecs", "warps", "set", "look"]
SHAPES = [(3136, 256, 2048), (3136, 256, 256), (12544, 64, 256), (2097152, 32, 4), (3025, 95, 64), (784, 512, 128), (8191, 3, 3),
          (1024, 5, 77), (65543, 3, 1), (512, 7, 4096), (163, 5, 300), (1100, 64, 33), (3136, 2, 1), (16, 3, 9)]


def keep(shape, direction, residual, tile, warp):
    out = (ctypes.c_uint32 * 10)()
    assert _lib.load().anode_gpu_batch_norm_tiled_keep(*shape, direction, residual, tile, warp, out) == 0
    return dict(zip(FIELDS, out))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("direction", [0, 1])
@pytest.mark.parametrize("residual", [0, 1])
def test_places_of_kept_tiles(shape, direction, residual):
    first = keep(shape, direction, residual, 0, 0)
    if not first["slots"]:
        return
    warps, vecs, look, columns = first["warps"], first["vecs"], first["look"], first["set"]
    room = 512 // (warps // 4)
    assert first["slots"] <= look + 1 and columns == 4 * (direction + 1)
    ranges = []                                   # per tile: the columns of every warp, or None
    kept_so_far = 0
    for t in range(2 * (look + 1) + 1):
        k = [keep(shape, direction, residual, t, w) for w in range(warps)]
        assert k[0]["before"] == kept_so_far
        kept_so_far += k[0]["kept"]
        if not k[0]["kept"]:
            ranges.append(None)
            continue
        assert sorted(v["dealt"] for v in k) == list(range(warps))
        mine = []
        for v in k:
            sets = max(0, -(-(vecs - 32 * v["dealt"]) // (32 * warps)))
            mine.append((v["column"], v["column"] + sets * columns))
            assert mine[-1][1] <= room
        ranges.append(mine)
    for t, mine in enumerate(ranges):             # tile t is written before tile t - look has been read
        for u in range(max(0, t - look), t):
            if mine and ranges[u]:
                for (a, b), (c, d) in zip(mine, ranges[u]):
                    assert b <= c or d <= a, (t, u)
    # evenly spread: as many of any period's tiles as there are places
    assert sum(r is not None for r in ranges[:look + 1]) == first["slots"]


def test_small_layers_have_no_smaller_tiles_for_a_larger_slot():
    """Forward pass of the residual epilogue: where the planner halves the tiles for want of enough of them, what it makes of the
    larger slots may be less than what it makes of smaller ones."""
    for shape, vectors in (((2888, 5, 149), 1444), ((2886, 5, 149), 1446), ((1197, 7, 94), 600), ((1364, 15, 113), 1364),
                           ((3136, 256, 256), 2352), ((3025, 95, 64), 2271)):
        assert keep(shape, 0, 1, 0, 0)["vecs"] == vectors, shape


def test_long_ragged_rows_of_the_residual_forward_pass_keep_no_tiles():
    for d0, forward in ((637, True), (639, True), (640, True), (641, False), (643, False), (6374, False), (6376, True)):
        shape = (d0, 20, 300)
        assert [bool(keep(shape, d, 1, 0, 0)["slots"]) for d in (0, 1)] == [forward, True], d0
        assert all(keep(shape, d, 0, 0, 0)["slots"] for d in (0, 1)), d0


def test_long_ragged_rows_of_the_forward_pass_keep_no_tiles():
    """Ordinary layers: from 24 channels on, where L2 keeps what lies between a tile's two visits; backward passes keep theirs."""
    for d0, c, n, forward in ((639, 95, 300, True), (641, 95, 300, False), (644, 95, 300, True), (3025, 95, 64, False), (3025, 23, 64, True),
                              (3025, 24, 64, False), (7485, 30, 1252, True)):
        assert [bool(keep((d0, c, n), d, 0, 0, 0)["slots"]) for d in (0, 1)] == [forward, True], (d0, c, n)
