"""Inference on a single large sample, whose rows are cut into pieces: in four, eight, five, three, seven and two, 16-byte loads and
4-byte ones, rows that cannot be cut, tensors off the 16-byte boundary; against torch in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c,row,offset", [(3, 1 << 19, 0), (96, 128 * 128, 0), (301, 5004, 0), (301, 5020, 0), (331, 4532, 0), (7, 221237, 0), (5, 3 * 100003, 0),
                                          (160, 16605, 0), (97, 128 * 128, 1), (30, 4 * 13003, 0), (30, 8 * 6503, 1), (2, 1000003, 0)])
def test_a_single_sample(c, row, offset):
    from anode_b200 import ops
    g = torch.Generator("cuda").manual_seed(c + row)
    buffers = [torch.randn(c * row + 4, device="cuda", generator=g) for _ in range(2)]
    x, y = (b[offset:offset + c * row].view(1, c, 1, row) for b in buffers)
    mean, var = torch.randn(c, device="cuda", generator=g), torch.rand(c, device="cuda", generator=g) * 3 + 0.5
    gamma, beta = torch.rand(c, device="cuda", generator=g) + 0.5, torch.randn(c, device="cuda", generator=g)
    ops.BatchNormalize2dActInferOp.apply([0, 1], x, mean, var, y, gamma, beta, 0.1)
    v = lambda t: t.double().view(1, c, 1, 1)
    t = (x.double() - v(mean)) / v(var).sqrt() * v(gamma) + v(beta)
    want = torch.where(t > 0, t, 0.1 * t)
    # four roundings of a value's parts, each within 2^-23 of the largest of them
    bound = 4 * 2.0 ** -23 * ((x.double().abs() + v(mean).abs()) / v(var).sqrt() * v(gamma) + v(beta).abs())
    assert ((y.double() - want).abs() <= bound).all()
