"""The ReLU and its adjoint at lengths where the kernel's split has remainders: less than a vector, whole vectors and a tail of one
to three floats, less and more than what the threads have in flight; in place, and off the 16-byte boundary.  Bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu

TURN = 148 * 64 * 256 * 4 * 4          # floats that the largest grid has in flight
LENGTHS = [1, 2, 3, 4, 5, 127, 1023, 1024, 1025, 256 * 4 * 2 * 148 - 1, 256 * 4 * 2 * 148, 256 * 4 * 4 * 2 * 148 + 3, 6422529, TURN - 1, TURN + 6]


@pytest.mark.parametrize("length", LENGTHS)
@pytest.mark.parametrize("offset", [0, 1])
def test_relu_and_its_adjoint(length, offset):
    from anode_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(length)

    def tensor():
        return torch.randn(length + offset, device="cuda", generator=g)[offset:]
    x, dy = tensor(), tensor()
    x[length // 2] = float("nan")
    guard = torch.full((length + offset + 8,), 7.0, device="cuda")
    y = guard[offset:offset + length]
    want = x * (x > 0)
    assert torch.equal(torch.nan_to_num(ops.PositiveClipOp.apply(x, y), nan=9.0), torch.nan_to_num(want, nan=9.0))
    assert (guard[offset + length:] == 7.0).all() and (guard[:offset] == 7.0).all()
    dz = guard[offset:offset + length]
    ops.PositiveClipBwdOp.apply(dy, x, dz)
    assert torch.equal(dz, dy * (x > 0))
    ops.relu(x, inplace=True)
    assert torch.equal(torch.nan_to_num(x, nan=9.0), torch.nan_to_num(want, nan=9.0))
