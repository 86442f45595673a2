"""The kernel for long rows, forced, is the one that each of the four calls launches: forward, backward and both of the residual epilogue."""
import numpy as np
import pytest
import torch

from tests.test_gpu_long import SHAPES, flat
from tests.util import make_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", SHAPES + [(4, 260, 1, 16384)])
def test_each_call(shape):
    from anode_b200 import ops
    shape = flat(shape)
    d = make_inputs(shape, seed=sum(shape), loc=3.0, scale=2.0)
    x, dy = torch.from_numpy(d["x"]).cuda(), torch.from_numpy(d["dy"]).cuda()
    c, op = shape[1], ops.BatchNormalize2dAddActFusedOp
    z = lambda: torch.zeros(c, device="cuda")
    mean, var, rm, rv, dg, db, y, dx, dr = z(), z(), z(), z(), z(), z(), torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    ws = ops.Workspace(*ops.dims_of(x), x.device)
    ops.set_kernel("long")
    try:
        for call in (lambda: ops.BatchNormalize2dFusedOp.apply([0, 1], 1e-5, 0.1, x, y, mean, var, rm, rv, None, None, workspace=ws, neg_slope=0.1),
                     lambda: ops.BatchNormalize2dBwdFusedOp.apply([0, 1], dy, x, mean, var, dx, None, None, dg, db, workspace=ws, neg_slope=0.1),
                     lambda: op.apply([0, 1], 1e-5, 0.1, x, dy, y, mean, var, rm, rv, None, None, 0.1, ws),
                     lambda: op.adjoint([0, 1], dy, x, y, mean, var, dx, dr, None, None, dg, db, 0.1, workspace=ws)):
            call()
            assert ops.last_kernel() == "long"
    finally:
        ops.set_kernel("auto")
    assert ws.status() == 0 and all(np.isfinite(t.cpu().numpy()).all() for t in (y, dx, dr))
