"""1/sqrt(variance + epsilon) as the kernels have it, seen through inference on x = 1 with mean 0 and no scale, where y is that value: the
lowest bit set, and one of the odd floats beside the exact value.  Odd floats lie two units apart, so the nearer one is at most one
unit of the last place off; the value that it is chosen from is rounded once and off by less than a hundredth beyond that."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def inv_std(v):
    from anode_b200 import ops
    c = v.numel()
    x, y = torch.ones(1, c, 1, 4, device="cuda"), torch.empty(1, c, 1, 4, device="cuda")
    ops.BatchNormalize2dActInferOp.apply([0, 1], x, torch.zeros(c, device="cuda"), v, y, None, None, 0.0)
    assert torch.equal(y.isnan(), y[..., :1].isnan().expand_as(y)) and bool(((y == y[..., :1]) | y.isnan()).all())
    return y[0, :, 0, 0].contiguous()


def variances():
    rng = np.random.default_rng(7)
    exponents = np.arange(-126, 128)
    mantissas = np.concatenate([1.0 + np.arange(8) * 2.0 ** -23, 2.0 - np.arange(1, 9) * 2.0 ** -23, 1.5 + np.arange(-3, 4) * 2.0 ** -23])
    edges = (mantissas[None] * 2.0 ** exponents[:, None]).ravel()
    spread = rng.uniform(1.0, 2.0, 200000) * 2.0 ** rng.integers(-126, 128, 200000)
    usual = rng.uniform(1e-5, 100.0, 200000)
    small = rng.integers(1, 1 << 23, 20000) * 2.0 ** -149                   # subnormal
    squares = (1.0 / rng.integers(1, 4000, 4000) ** 2.0)
    return np.concatenate([edges, spread, usual, small, squares]).astype(np.float32)


def test_the_nearer_odd_value():
    v = variances()
    got = inv_std(torch.from_numpy(v).cuda()).cpu().numpy()
    want = 1.0 / np.sqrt(v.astype(np.float64))
    unit = 2.0 ** (np.floor(np.log2(want)) - 23)
    assert (got.view(np.uint32) & 1 == 1).all()
    assert (np.abs(got.astype(np.float64) - want) <= 1.01 * unit).all()


def test_zero_infinity_nan_and_below_zero():
    got = inv_std(torch.tensor([0.0, float("inf"), float("nan"), -1.0, 1.0], device="cuda")).cpu().numpy()
    assert np.isnan(got[[0, 2, 3]]).all() and got.view(np.uint32)[1] == 1 and abs(got[4] - 1.0) <= 2.0 ** -23
    assert (got.view(np.uint32) & 1 == 1)[[1, 4]].all()
