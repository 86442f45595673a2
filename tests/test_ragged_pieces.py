"""Ragged rows that the tiled kernel cuts into pieces: none may hold fewer than four floats, since a 16-byte vector of it is then
taken for one that lies wholly within it (no GPU needed)."""
import random

import pytest
import torch

from anode_b200 import _lib, ops

#: shapes whose pieces of an even size would leave one of one to three floats, in the forward or the backward pass
SHORT = [(1, 1, 511, 511), (2, 1, 511, 511), (1, 2, 511, 511), (1, 1, 513, 513), (1, 1, 589, 589), (1, 1, 1023, 1023)]


def last_pieces(d0, c, n):
    return [_lib.load().anode_gpu_batch_norm_tiled_last_piece(d0, c, n, direction, residual) for direction in (0, 1) for residual in (0, 1)]


@pytest.mark.parametrize("shape", SHORT)
def test_shapes_that_were_cut_short(shape):
    pieces = last_pieces(*ops.dims_of(torch.empty(shape, device="meta")))
    assert all(p >= 4 for p in pieces), pieces
    assert [ops.serving_kernel(shape, direction) for direction in (0, 1)] == ["tiled", "tiled"]


def test_no_piece_of_fewer_than_four_floats():
    rng = random.Random(1)
    rows = list(range(1001, 40000, 14)) + [rng.randrange(40000, 4000000) for _ in range(4000)] + [4091 * 4091, 16777217, 2 ** 27 + 1]
    cut = 0
    for d0 in rows:
        for c, n in ((1, 1), (2, 1), (3, 5), (95, 2)):
            if d0 * c * n >= 1 << 32:
                continue
            pieces = last_pieces(d0, c, n)
            assert all(p >= 4 for p in pieces if p), (d0, c, n, pieces)
            cut += sum(0 < p < d0 for p in pieces)
    assert cut > 10000
