"""Accumulating input gradients (WriteCap.Accumulate) on every kernel: what was there plus what the assigning call writes, to the bit.
Tiles, batches and rows with remainders, rows that begin anywhere, tensors that end inside a 16-byte vector."""
import pytest
import torch

from tests.util import make_inputs

pytestmark = pytest.mark.gpu

CASES = [("tiled", (64, 8, 56, 56)), ("tiled", (40, 24, 36, 36)), ("tiled", (9, 5, 55, 55)), ("tiled", (700, 3, 33, 31)), ("tiled", (3, 3, 161, 121)),
         ("band", (1283, 244, 7, 7)), ("band", (700, 4500, 1, 5)), ("band", (60, 1004, 16, 17)), ("stream", (1411, 128, 7, 7)), ("stream", (301, 13, 5, 5)),
         ("long", (13, 6, 1, 3001)), ("long", (64, 8, 56, 56)), ("register", (5, 3, 7, 7)), ("register", (64, 300, 7, 7)), ("register", (15, 64, 28, 28)),
         ("plain", (64, 8, 56, 56))]


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("kernel,shape", CASES)
def test_adds_what_the_assigning_call_writes(kernel, shape, residual):
    from anode_b200 import ops
    d = make_inputs(shape, seed=sum(shape), loc=0.5, scale=2.0)
    t = {k: None if v is None else torch.from_numpy(v).cuda() for k, v in d.items()}
    x, dy, c = t["x"], t["dy"], shape[1]
    old = torch.randn(shape, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    mean, var = x.mean((0, 2, 3)), x.var((0, 2, 3), unbiased=False) + 1e-5
    got = []
    ops.set_kernel(kernel)
    try:
        for cap in (ops.WriteCap.Assign, ops.WriteCap.Accumulate):
            dx, dg, db = old.clone(), torch.zeros(c, device="cuda"), torch.zeros(c, device="cuda")
            ws = ops.Workspace(*ops.dims_of(x), x.device)
            if residual:
                dres = torch.empty_like(x)
                ops.BatchNormalize2dAddActFusedOp.adjoint([0, 1], dy, x, x, mean, var, dx, dres, t["gamma"], t["beta"], dg, db, 0.1, cap=cap, workspace=ws)
            else:
                dres = None
                ops.BatchNormalize2dBwdFusedOp.apply([0, 1], dy, x, mean, var, dx, t["gamma"], t["beta"], dg, db, cap=cap, workspace=ws, neg_slope=0.1)
            assert ops.last_kernel() == kernel and ws.status() == 0
            got.append((dx, dg, db, dres))
    finally:
        ops.set_kernel("auto")
    assert torch.equal(got[1][0], old + got[0][0])
    assert torch.equal(got[1][1], got[0][1]) and torch.equal(got[1][2], got[0][2])
    assert not residual or torch.equal(got[1][3], got[0][3])
