"""Ragged rows that the tiled kernel cuts into pieces of which the last holds one to three floats: which vectors count as lying
wholly within a piece, and which shapes have such a piece (no GPU needed)."""
import ctypes

import pytest
import torch

from anode_b200 import _lib, ops

#: shape, and the directions in which its last piece is that short
SHORT = [((1, 1, 511, 511), (0, 1)), ((2, 1, 511, 511), (0,)), ((1, 2, 511, 511), (0,)), ((1, 1, 513, 513), (0, 1)),
         ((1, 1, 589, 589), (1,)), ((1, 1, 1023, 1023), (0,))]


@pytest.mark.parametrize("length", list(range(1, 14)) + [1021, 65531])
def test_a_whole_vector_lies_within_its_piece(length):
    whole = _lib.load().anode_gpu_batch_norm_ragged_whole
    for first in list(range(-3, min(length, 20) + 5)) + list(range(max(0, length - 9), length + 5)):
        assert whole(first, length) == int(first >= 0 and first + 4 <= length), (first, length)
    assert whole(length, length) == 0            # how a missing vector is described


@pytest.mark.parametrize("shape,directions", SHORT)
def test_shapes_with_a_short_last_piece(shape, directions):
    for direction in directions:
        out = (ctypes.c_uint32 * 12)()
        d0, c, n = ops.dims_of(torch.empty(shape, device="meta"))
        assert _lib.load().anode_gpu_batch_norm_tiled_geometry(d0, c, n, direction, out) == 0
        assert out[0] and 1 <= d0 % out[2] <= 3, list(out)
        assert ops.serving_kernel(shape, direction) == "tiled"
