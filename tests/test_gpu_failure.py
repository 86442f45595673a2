"""Failure detection on the device, in the form that cannot hurt a GPU: a synchronized call whose peer
never writes its records.  One process, one GPU, an exchange-only communicator that claims two ranks
with both exchange buffers in local memory; the wait limit is set to 20 ms, so the kernel's bounded
wait runs out, the status word says so, the kernel drains and returns, and after a re-initialisation
the same workspace serves a normal call.  Nothing here faults, traps or spins without bound."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import bn_oracle as o
from tests.util import check_layer, make_inputs

pytestmark = pytest.mark.gpu

WAIT_STATS, WAIT_PEER, ABORTED = 1, 2, 4


@pytest.fixture
def short_waits():
    from anode_b200 import ops
    ops.set_wait_limit_ms(20)
    yield ops
    ops.set_wait_limit_ms(1500)
    ops.set_kernel("auto")


@pytest.mark.parametrize("kernel,shape", [("tiled", (16, 8, 56, 56)), ("resident", (16, 8, 56, 56)), ("cluster", (32, 64, 7, 7)),
                                          ("plain", (6, 3, 5, 5))])
def test_wait_for_an_absent_peer_runs_out_and_the_workspace_recovers(short_waits, kernel, shape):
    ops = short_waits
    from anode_b200 import _lib, sync
    lib = _lib.load()
    ops.set_kernel(kernel)
    d = make_inputs(shape, seed=81, loc=0.5, scale=2.0)
    x = torch.from_numpy(d["x"]).cuda(); dy = torch.from_numpy(d["dy"]).cuda()
    c = shape[1]
    comm = sync.SyncComm.exchange_only(0, 2)
    nbytes = int(lib.anode_gpu_sync_exchange_bytes(c, 2))
    bufs = [torch.zeros(nbytes, dtype=torch.uint8, device="cuda") for _ in range(2)]
    comm.attach_exchange_pointers(bufs, c)
    layer = ops.SyncBatchNormRelu(c, comm=comm, global_count=2 * x.numel() // c)
    layer.gamma.copy_(torch.from_numpy(d["gamma"])); layer.beta.copy_(torch.from_numpy(d["beta"]))
    t0 = torch.cuda.Event(enable_timing=True); t1 = torch.cuda.Event(enable_timing=True)
    t0.record()
    layer.forward(x)
    t1.record()
    torch.cuda.synchronize()
    status = layer.status()
    assert status & WAIT_PEER, status
    if kernel in ("tiled", "resident"):
        assert status & ABORTED, status
    assert t0.elapsed_time(t1) < 1000.0          # the 20 ms bound, not the default 1.5 s, and certainly no hang
    # this rank's own record did reach "the peer" (a local buffer here): the exchange itself works
    assert int(bufs[1].view(torch.int64).ne(0).sum()) > 0
    comm.destroy()
    # recovery: re-initialise the workspace, then a normal (one-GPU) call on it is right again
    ops.set_wait_limit_ms(1500)
    ws = layer._ws
    ws.reset()
    torch.cuda.synchronize()
    assert ws.status() == 0
    mean = torch.zeros(c, device="cuda"); var = torch.zeros(c, device="cuda")
    rm = torch.from_numpy(d["run_mean"]).cuda(); rv = torch.from_numpy(d["run_var"]).cuda()
    dg = torch.zeros(c, device="cuda"); db = torch.zeros(c, device="cuda")
    y = torch.empty_like(x); dx = torch.empty_like(x)
    axes = list(range(x.dim() - 2))
    ops.BatchNormalize2dFusedOp.apply(axes, 1e-5, 0.1, x, y, mean, var, rm, rv, layer.gamma, layer.beta, True, ws)
    ops.BatchNormalize2dBwdFusedOp.apply(axes, dy, x, mean, var, dx, layer.gamma, layer.beta, dg, db, True, ops.WriteCap.Assign, ws)
    torch.cuda.synchronize()
    assert ws.status() == 0
    got = dict(y=y.cpu().numpy(), dx=dx.cpu().numpy(), mean=mean.cpu().numpy(), var=var.cpu().numpy(), run_mean=rm.cpu().numpy(),
               run_var=rv.cpu().numpy(), dgamma=dg.cpu().numpy(), dbeta=db.cpu().numpy())
    truth = o.bn_relu_fwd_bwd_f64(d["x"], d["dy"], 1e-5, 0.1, d["run_mean"], d["run_var"], d["gamma"], d["beta"])
    check_layer(got, truth, d["x"], d["gamma"], d["beta"], "after recovery ")


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("kernel,shape", [("band", (1283, 244, 7, 7)), ("band", (256, 512, 14, 14)), ("tiled", (64, 95, 55, 55)),
                                          ("tiled", (64, 64, 56, 56))])
def test_a_wait_that_runs_out_leaves_no_copy_and_no_state_behind(kernel, shape, residual):
    """A bound of one cycle: the first poll for a channel's words finds none, in every block, with copies on their way into the
    slots.  The call says so, returns at once (the default bound is 1.5 s), and after a re-initialisation the workspace serves."""
    from anode_b200 import _lib, ops
    from tests.test_gpu_band import inputs, run
    d = inputs(shape, 3)
    c, x = shape[1], d["x"]
    ops.set_kernel(kernel)
    try:
        want, ws = run(ops, d, residual, 0.1, launched=kernel)
        z = [torch.zeros(c, device="cuda") for _ in range(4)]
        y, dx, dres = (torch.empty_like(x) for _ in range(3))
        if residual:
            op = ops.BatchNormalize2dAddActFusedOp
            calls = [lambda: op.apply([0, 1], 1e-5, 0.1, x, d["res"], y, z[0], z[1], z[2], z[3], d["gamma"], d["beta"], 0.1, ws),
                     lambda: op.adjoint([0, 1], d["dy"], x, want["y"], want["mean"], want["var"], dx, dres, d["gamma"], d["beta"], z[0], z[1], 0.1,
                                        workspace=ws)]
        else:
            calls = [lambda: ops.BatchNormalize2dFusedOp.apply([0, 1], 1e-5, 0.1, x, y, z[0], z[1], z[2], z[3], d["gamma"], d["beta"], workspace=ws, neg_slope=0.1),
                     lambda: ops.BatchNormalize2dBwdFusedOp.apply([0, 1], d["dy"], x, want["mean"], want["var"], dx, d["gamma"], d["beta"], z[0], z[1],
                                                                  workspace=ws, neg_slope=0.1)]
        for call in calls:
            t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            assert _lib.load().anode_gpu_batch_norm_fused_set_wait_limit_cycles(1) == 0
            t0.record()
            call()
            t1.record()
            torch.cuda.synchronize()
            ops.set_wait_limit_ms(1500)
            assert ws.status() == WAIT_STATS | ABORTED
            assert t0.elapsed_time(t1) < 500.0
            ws.reset()
        for _ in range(2):
            again, _ = run(ops, d, residual, 0.1, ws, launched=kernel)
            assert all(torch.equal(again[k], want[k]) for k in want)
    finally:
        ops.set_wait_limit_ms(1500)
        ops.set_kernel("auto")


def test_the_wait_limit_is_never_nothing():
    from anode_b200 import _lib
    lib = _lib.load()
    assert lib.anode_gpu_batch_norm_fused_set_wait_limit_ms(0) == -2 and lib.anode_gpu_batch_norm_fused_set_wait_limit_cycles(0) == -2      # ANODE_E_DIMS


def test_exchange_only_communicator_refuses_what_it_cannot_do():
    from anode_b200 import _lib, sync
    lib = _lib.load()
    comm = sync.SyncComm.exchange_only(1, 2)
    buf = torch.zeros(8, device="cuda")
    # no NCCL behind it: the gradient all-reduce is refused, nothing is enqueued
    assert lib.anode_gpu_sync_allreduce_sum_f32(comm.handle, ctypes.c_void_p(buf.data_ptr()), 8, None) == -5
    # no exchange attached yet: a synchronized call is refused as well
    ws = torch.zeros(int(lib.anode_gpu_sync_batch_norm_workspace_bytes(64, 4, 2, 2)), dtype=torch.uint8, device="cuda")
    x = torch.zeros(2, 4, 8, 8, device="cuda"); v = torch.zeros(4, device="cuda")
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = lib.anode_gpu_sync_batch_norm_relu_fwd_3d1_packed_f32(64, 4, 2, 1e-5, 0.1, 1, p(x), None, None, p(x), p(v), p(v), None, None,
                                                               comm.handle, p(ws), ws.numel(), None, None)
    assert rc == -5
    torch.cuda.synchronize()
    comm.destroy()
