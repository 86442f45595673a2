"""The band kernel at the sizes where its splits have remainders: a last unit of fewer channels, a last tile of fewer samples,
vectors shared by two channels, one sample group and many, one box and several, the most channels of a unit; the residual
epilogue, outputs over inputs, a channel with a NaN or an infinity, and other kernels between its launches on one workspace.  Every call is
asserted to have launched it: where the device refuses it, the streaming kernel serves."""
import ctypes

import pytest
import torch

from tests.test_band_plan import band
from tests.test_gpu_tiled_forms import outputs_over_inputs

pytestmark = pytest.mark.gpu

SHAPES = [(1283, 244, 7, 7), (300, 257, 14, 14), (500, 2003, 4, 4), (1999, 64, 11, 11), (81, 900, 15, 15), (1000, 2602, 2, 3), (60, 1004, 16, 17),
          (1024, 250, 8, 8), (333, 1000, 7, 7), (801, 5002, 2, 2), (700, 4500, 1, 5),
          (1351, 244, 7, 7), (2481, 128, 7, 7)]         # a last tile of one sample: groups without any


@pytest.fixture
def forced():
    from anode_b200 import ops
    ops.set_kernel("band")
    yield ops
    ops.set_kernel("auto")


def inputs(shape, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    c = shape[1]
    x = torch.randn(shape, device="cuda", generator=g) * 2 + 3 * torch.rand(1, c, 1, 1, device="cuda", generator=g)
    return dict(x=x, dy=torch.randn(shape, device="cuda", generator=g), res=torch.randn(shape, device="cuda", generator=g),
                gamma=torch.rand(c, device="cuda", generator=g) + 0.5, beta=torch.rand(c, device="cuda", generator=g) * 0.2 - 0.1)


def run(ops, d, residual, slope, ws=None, launched="band"):
    """Forward and backward call, each launched by the kernel of that name (None: by any)."""
    def check_kernel():
        assert launched is None or ops.last_kernel() == launched, (tuple(d["x"].shape), ops.last_kernel())
    x, c = d["x"], d["x"].shape[1]
    z = lambda: torch.zeros(c, device="cuda")
    r = dict(mean=z(), var=z(), run_mean=z(), run_var=z() + 1, dgamma=z(), dbeta=z(), y=torch.full_like(x, float("nan")), dx=torch.full_like(x, float("nan")))
    ws = ws or ops.Workspace(*ops.dims_of(x), x.device)
    if residual:
        r["dres"] = torch.full_like(x, float("nan"))
        op = ops.BatchNormalize2dAddActFusedOp
        op.apply([0, 1], 1e-5, 0.1, x, d["res"], r["y"], r["mean"], r["var"], r["run_mean"], r["run_var"], d["gamma"], d["beta"], slope, ws)
        check_kernel()
        op.adjoint([0, 1], d["dy"], x, r["y"], r["mean"], r["var"], r["dx"], r["dres"], d["gamma"], d["beta"], r["dgamma"], r["dbeta"], slope, workspace=ws)
    else:
        ops.BatchNormalize2dFusedOp.apply([0, 1], 1e-5, 0.1, x, r["y"], r["mean"], r["var"], r["run_mean"], r["run_var"], d["gamma"], d["beta"],
                                          workspace=ws, neg_slope=slope)
        check_kernel()
        ops.BatchNormalize2dBwdFusedOp.apply([0, 1], d["dy"], x, r["mean"], r["var"], r["dx"], d["gamma"], d["beta"], r["dgamma"], r["dbeta"],
                                             workspace=ws, neg_slope=slope)
    check_kernel()
    assert ws.status() == 0
    return r, ws


def check(d, got, residual, slope, what):
    """Against float64 with the layer's own activation decisions, exact ones away from zero; the tolerance of tests/util.py."""
    x, dy = d["x"].double(), d["dy"].double()
    ax, m = (0, 2, 3), x.numel() // x.shape[1]
    v = lambda t: t.double().view(1, -1, 1, 1)
    mean, var = x.mean(ax), x.var(ax, unbiased=False) + 1e-5
    rstd = 1 / var.sqrt()
    xhat = (x - v(mean)) * v(rstd)
    pre = xhat * v(d["gamma"]) + v(d["beta"]) + (d["res"].double() if residual else 0)
    mask = got["y"] > 0
    assert not ((mask != (pre > 0)) & (pre.abs() >= 1e-5)).any(), what
    act = torch.where(mask, 1.0, slope).double()
    dz = dy * act
    s1, s2 = dz.sum(ax), (dz * xhat).sum(ax)
    want = dict(y=pre * act, mean=mean, var=var, run_mean=0.1 * mean, run_var=1 + 0.1 * (var - 1), dbeta=s1, dgamma=s2,
                dx=v(d["gamma"]) * v(rstd) * (dz - v(s1) / m - xhat * v(s2) / m))
    if residual:
        want["dres"] = dz
    for k, w in want.items():
        atol = 1e-5 + (1e-4 * float(w.square().mean().sqrt()) if k in ("dgamma", "dbeta") else 0.0)
        off = (got[k].double() - w).abs() > atol + 1e-4 * w.abs()
        assert not off.any(), (what, k, int(off.sum()), off.nonzero()[0].tolist())


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("residual", [False, True])
def test_against_float64(forced, shape, residual):
    ops = forced
    for direction in (0, 1):
        assert band(shape, direction, residual)["taken"] == 1 and ops.serving_kernel(shape, direction, residual=residual) == "stream"
    d, slope = inputs(shape, sum(shape)), 0.1 if shape[0] % 2 else 0.0
    got, ws = run(ops, d, residual, slope)
    check(d, got, residual, slope, shape)
    for _ in range(2):                           # the other buffer of words, and the first one again
        again, _ = run(ops, d, residual, slope, ws)
        assert all(torch.equal(again[k], got[k]) for k in got), shape


@pytest.mark.parametrize("form", ["dres is dy", "dres is y", "dres is x", "no dres", "dx is dy", "dx is x", "accumulate"])
def test_outputs_over_inputs(form):
    from anode_b200 import ops
    assert band((1411, 132, 7, 7), 1, 1)["taken"] == 1
    outputs_over_inputs(ops, (1411, 132, 7, 7), form, "band")
    assert ops.last_kernel() == "band"


def test_calls_without_what_is_optional(forced):
    """No gamma and beta, no averages, no gradients of gamma and beta, dx accumulated: the ordinary form and the residual epilogue."""
    ops, shape = forced, (1283, 244, 7, 7)
    d = inputs(shape, 6)
    c, x, dy = shape[1], d["x"], d["dy"]
    m = x.numel() // c
    v = lambda t: t.double().view(1, -1, 1, 1)
    ws = ops.Workspace(*ops.dims_of(x), x.device)
    launched = lambda: ops.last_kernel() == "band" or pytest.fail(str(ops.last_kernel()))
    for residual in (False, True):
        mean, var, y, dx = torch.zeros(c, device="cuda"), torch.zeros(c, device="cuda"), torch.empty_like(x), torch.ones_like(x)
        if residual:
            ops.BatchNormalize2dAddActFusedOp.apply([0, 1], 1e-5, 0.1, x, d["res"], y, mean, var, workspace=ws)
            launched()
            ops.BatchNormalize2dAddActFusedOp.adjoint([0, 1], dy, x, y, mean, var, dx, cap=ops.WriteCap.Accumulate, workspace=ws)
        else:
            ops.BatchNormalize2dFusedOp.apply([0, 1], 1e-5, 0.1, x, y, mean, var, workspace=ws)
            launched()
            ops.BatchNormalize2dBwdFusedOp.apply([0, 1], dy, x, mean, var, dx, cap=ops.WriteCap.Accumulate, workspace=ws)
        launched()
        assert ws.status() == 0
        xhat = (x.double() - v(x.double().mean((0, 2, 3)))) / v((x.double().var((0, 2, 3), unbiased=False) + 1e-5).sqrt())
        pre = xhat + (d["res"].double() if residual else 0)
        mask = y > 0
        assert not ((mask != (pre > 0)) & (pre.abs() >= 1e-5)).any()
        dz = dy.double() * mask
        want = 1 + (dz - v(dz.sum((0, 2, 3))) / m - xhat * v((dz * xhat).sum((0, 2, 3))) / m) / v(var.double().sqrt())
        for got, w in ((y, pre * mask), (dx, want)):      # the tolerance of tests/util.py
            assert not ((got.double() - w).abs() > 1e-5 + 1e-4 * w.abs()).any(), residual


def test_other_kernels_between_its_launches_on_one_workspace(forced):
    ops, shape = forced, (1283, 244, 7, 7)
    d = inputs(shape, 7)
    want, ws = run(ops, d, False, 0.0)
    want_res, _ = run(ops, d, True, 0.0, ws)
    for kernel in ("plain", "auto", "register", "stream"):
        ops.set_kernel(kernel)
        check(d, run(ops, d, False, 0.0, ws, launched="band" if kernel == "auto" else kernel)[0], False, 0.0, kernel)
        ops.set_kernel("band")
        for residual, w in ((False, want), (True, want_res)):
            got, _ = run(ops, d, residual, 0.0, ws)
            assert all(torch.equal(got[k], w[k]) for k in w), (kernel, residual)


def test_a_poisoned_channel_has_no_variance(forced):
    ops, shape = forced, (1283, 244, 7, 7)
    d = inputs(shape, 8)
    clean, _ = run(ops, d, False, 0.0)
    for place in (0, 777):
        x = d["x"].clone()
        x[place, 0, 3, 2], x[place, 2, 6, 6] = float("nan"), float("inf")
        got, _ = run(ops, dict(d, x=x), False, 0.0)
        for c in (0, 2):
            assert torch.isnan(got["var"][c]) and torch.isnan(got["run_var"][c]) and not torch.isfinite(got["mean"][c])
            assert torch.isnan(got["y"][:, c]).all()
        assert got["mean"][2] == float("inf")
        rest = [c for c in range(shape[1]) if c not in (0, 2)]
        for k in ("mean", "var", "run_mean", "run_var", "dgamma", "dbeta"):
            assert torch.equal(got[k][rest], clean[k][rest]), k
        for k in ("y", "dx"):
            assert torch.equal(got[k][:, rest], clean[k][:, rest]), k


def test_means_far_from_zero_keep_the_variances_digits(forced):
    """The shift of a thread's sums comes from four of its samples in each tile; with the mean at 300 standard deviations the
    bound is that of the inputs' own rounding, 2^-24 * 300 relative to a deviation, for the mean of a few thousand of them."""
    ops, shape = forced, (1024, 320, 7, 7)
    d = inputs(shape, 9)
    d["x"] = torch.randn(shape, device="cuda") + 300.0
    got, _ = run(ops, d, False, 0.0)
    x = d["x"].double()
    var = x.var((0, 2, 3), unbiased=False) + 1e-5
    assert float(((got["var"].double() - var) / var).abs().max()) < 300 * 2.0 ** -24
    assert float((got["mean"].double() - x.mean((0, 2, 3))).abs().max()) < 300 * 2.0 ** -23


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("shape", [(1024, 320, 7, 7), (1283, 244, 7, 7), (300, 257, 14, 14), (1999, 64, 11, 11), (700, 4500, 1, 5), (500, 2003, 4, 4)])
def test_sums_are_rounded_once(forced, shape, residual):
    """Whole numbers, such that what a thread adds up in f32 is exact (forward: squares of quarters below 256, 16 of them, are sixteenths below
    2^20; backward: 8 numbers below 2^20): the results are the exact sums, rounded once to f32, 2^-24 relative.  (No last tile here leaves a
    thread with three samples, whose mean is no shift in quarters.)"""
    ops = forced
    for direction in (0, 1):
        assert band(shape, direction, residual)["taken"] == 1
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(shape))
    c, n = shape[1], shape[0] * shape[2] * shape[3]
    ints = lambda low, high: torch.randint(low, high, shape, device="cuda", generator=g).float()
    z = lambda: torch.zeros(c, device="cuda")
    x = ints(-100, 101) + torch.randint(-50, 51, (1, c, 1, 1), device="cuda", generator=g).float()
    y, mean, var = torch.empty_like(x), z(), z()
    ws = ops.Workspace(*ops.dims_of(x), x.device)
    if residual:
        ops.BatchNormalize2dAddActFusedOp.apply([0, 1], 1e-5, 0.1, x, x, y, mean, var, z(), z(), None, None, 1.0, ws)
    else:
        ops.BatchNormalize2dFusedOp.apply([0, 1], 1e-5, 0.1, x, y, mean, var, z(), z(), None, None, workspace=ws, neg_slope=1.0)
    ax = (0, 2, 3)
    s1, s2 = x.double().sum(ax), x.double().square().sum(ax)
    epsilon = float(torch.tensor(1e-5))
    once = lambda got, want, what: float(((got.double() - want).abs() - 2.0 ** -24 * (1 + 1e-6) * want.abs()).max()) <= 0 or pytest.fail(what)
    once(mean, s1 / n, "mean")
    once(var, (s2 - s1 * s1 / n) / n + epsilon, "var")
    # about a mean of zero and with a variance of one, whose 1 / std has its lowest bit set (inv_std): dgamma is sum(dz * x), with x of -1, 0, 1
    x, dy = ints(-1, 2), ints(-(2 ** 20) + 1, 2 ** 20)
    dx, dgamma, dbeta = torch.empty_like(x), z(), z()
    if residual:
        ops.BatchNormalize2dAddActFusedOp.adjoint([0, 1], dy, x, y, z(), z() + 1, dx, torch.empty_like(x), None, None, dgamma, dbeta, 1.0, workspace=ws)
    else:
        ops.BatchNormalize2dBwdFusedOp.apply([0, 1], dy, x, z(), z() + 1, dx, None, None, dgamma, dbeta, workspace=ws, neg_slope=1.0)
    assert ws.status() == 0
    once(dbeta, dy.double().sum(ax), "dbeta")
    once(dgamma, (dy.double() * x.double()).sum(ax) * (1 + 2.0 ** -23), "dgamma")
