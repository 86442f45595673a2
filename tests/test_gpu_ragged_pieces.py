"""The tiled kernel on ragged rows whose pieces are cut so that the last one holds four floats or more
(tests/test_ragged_pieces.py): results against float64, and not a float written outside y, dx and dresidual."""
import numpy as np
import pytest
import torch

from tests.test_gpu_fused import dev, host
from tests.test_ragged_pieces import SHORT
from tests.util import check_layer_own_mask, make_inputs

pytestmark = pytest.mark.gpu

GUARD = 8           # floats before and behind an output


def guarded(shape, fill):
    size = int(np.prod(shape))
    a = torch.full((size + 2 * GUARD,), 7.0, device="cuda")
    t = a[GUARD:GUARD + size].view(shape)
    t.fill_(fill)
    return a, t


@pytest.mark.parametrize("shape", SHORT)
@pytest.mark.parametrize("residual", [False, True])
def test_short_last_pieces(shape, residual):
    from anode_b200 import ops
    d = make_inputs(shape, seed=sum(shape), loc=0.5, scale=2.0)
    res = np.random.default_rng(5).standard_normal(shape).astype(np.float32)
    t = {k: dev(v) for k, v in d.items()}
    c, slope = shape[1], 0.1
    mean, var, dg, db = (torch.zeros(c, device="cuda") for _ in range(4))
    ws = ops.Workspace(*ops.dims_of(t["x"]), t["x"].device)
    ops.set_kernel("tiled")
    try:
        for accumulate in (False, True):
            (ya, y), (dxa, dx), (dra, dres) = guarded(shape, float("nan")), guarded(shape, 1.0 if accumulate else float("nan")), guarded(shape, float("nan"))
            kw = dict(workspace=ws, neg_slope=slope)
            cap = ops.WriteCap.Accumulate if accumulate else ops.WriteCap.Assign
            run_mean, run_var = t["run_mean"].clone(), t["run_var"].clone()
            if residual:
                op = ops.BatchNormalize2dAddActFusedOp
                op.apply([0, 1], 1e-5, 0.1, t["x"], dev(res), y, mean, var, run_mean, run_var, t["gamma"], t["beta"], **kw)
                op.adjoint([0, 1], t["dy"], t["x"], y, mean, var, dx, dres, t["gamma"], t["beta"], dg, db, cap=cap, **kw)
            else:
                ops.BatchNormalize2dFusedOp.apply([0, 1], 1e-5, 0.1, t["x"], y, mean, var, run_mean, run_var, t["gamma"], t["beta"], **kw)
                ops.BatchNormalize2dBwdFusedOp.apply([0, 1], t["dy"], t["x"], mean, var, dx, t["gamma"], t["beta"], dg, db, cap=cap, **kw)
            assert ws.status() == 0
            got = dict(y=host(y), dx=host(dx) - (1.0 if accumulate else 0.0), mean=host(mean), var=host(var), dgamma=host(dg), dbeta=host(db))
            if residual:
                got["dresidual"] = host(dres)
            # (an accumulated gradient is rounded as a sum with 1: at most 2^-22 for values below 8, far below the bound of 1e-5)
            check_layer_own_mask(d, got, "%r residual %d accumulate %d " % (shape, residual, accumulate),
                                 residual=res if residual else None, slope=slope)
            for name, a in (("y", ya), ("dx", dxa), ("dresidual", dra)):
                assert bool((a[:GUARD] == 7.0).all() and (a[-GUARD:] == 7.0).all()), name
    finally:
        ops.set_kernel("auto")
