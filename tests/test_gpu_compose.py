"""The one-launch composition and its adjoint (csrc/bn_compose.cu) against float64, op by op: channels held in registers by a
warp, a block and clusters, channels that are not, 16- and 4-byte loads, unaligned tensors, and a mean and variance that are
not the batch's."""
import numpy as np
import pytest
import torch

from anode_b200 import _lib, ops
from tests.test_gpu_fused import dev, host
from tests.util import assert_close, assert_sum_close, make_inputs

SHAPES = [(2, 3, 1, 1), (2, 5, 3, 3), (3, 2, 16, 16), (32, 4, 28, 28), (64, 3, 28, 28), (85, 3, 28, 28), (86, 3, 28, 28),
          (9, 5, 55, 55), (700, 3, 7, 7), (1, 2, 1, 16384), (1, 2, 1, 16385), (1, 2, 1, 65536), (1, 2, 1, 65540), (4, 3, 128, 200),
          (2, 2, 5, 6, 7), (600, 40, 2, 2)]


def address(name):
    return getattr(_lib.load(), name)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("offset", [0, 1])
def test_composition_and_adjoint(shape, offset):
    d = make_inputs(shape, seed=sum(shape), loc=0.5, scale=2.0, affine=False)
    c, ax = shape[1], tuple(i for i in range(len(shape)) if i != 1)
    bs = (1, c) + (1,) * (len(shape) - 2)
    axes = list(range(len(shape) - 2))

    def place(a):
        t = torch.empty(a.size + offset, device="cuda")[offset:].view(shape)
        return t.copy_(torch.from_numpy(a))
    x64, dy64 = d["x"].astype(np.float64), d["dy"].astype(np.float64)
    m = x64.size // c
    tx, tdy = place(d["x"]), place(d["dy"])
    am, av = dev(d["run_mean"]), dev(d["run_var"])
    want_mean, want_var = x64.mean(ax), x64.var(ax) + 1e-5
    for kernel in ("auto", "plain"):           # the fused calls' kernels where they serve, and this file's own
        ops.set_kernel(kernel)
        try:
            am, av = dev(d["run_mean"]), dev(d["run_var"])
            y, mean, var, am, av = ops.batch_normalize_2d(tx, axes, True, 0.1, 1e-5, am, av)
        finally:
            ops.set_kernel("auto")
        assert_close(host(mean), want_mean, "mean")
        assert_close(host(var), want_var, "var")
        assert_close(host(am), 0.1 * want_mean, "running mean")
        assert_close(host(av), 0.9 + 0.1 * want_var, "running variance")
        assert_close(host(y), (x64 - want_mean.reshape(bs)) / np.sqrt(want_var).reshape(bs), "y")
    # the adjoint at a mean and a variance of the caller's
    rng = np.random.default_rng(3)
    for mean32, var32 in ((want_mean.astype(np.float32), want_var.astype(np.float32)),
                          (rng.standard_normal(c).astype(np.float32), (rng.random(c) + 0.5).astype(np.float32))):
        dx, dmean, dvar = ops.batch_normalize_adjoint(axes, tdy, tx, dev(mean32), dev(var32))
        e = x64 - mean32.astype(np.float64).reshape(bs)
        r = 1.0 / np.sqrt(var32.astype(np.float64))
        wvar = (dy64 * e).sum(ax) * -0.5 * r / var32
        wmean = -r * dy64.sum(ax) - 2.0 * wvar * e.sum(ax) / m
        assert_sum_close(host(dvar), wvar, "dvar")
        assert_sum_close(host(dmean), wmean, "dmean")
        assert_close(host(dx), dy64 * r.reshape(bs) + (2.0 * wvar / m).reshape(bs) * e + (wmean / m).reshape(bs), "dx")


@pytest.mark.gpu
def test_arrays_without_elements_and_running_statistics_go_op_by_op():
    x = torch.empty(0, 3, 4, 4, device="cuda")
    y, mean, var, am, av = ops.batch_normalize_2d(x, [0, 1], True, 0.1, 1e-5)
    assert y.shape == x.shape and mean.tolist() == var.tolist() == am.tolist() == av.tolist() == [0.0] * 3
    dx, dmean, dvar = ops.batch_normalize_adjoint([0, 1], x, x, mean, var)
    assert dx.shape == x.shape and dmean.tolist() == dvar.tolist() == [0.0] * 3


def test_refusals():
    x, v = torch.zeros(2, 3, 4, 4), torch.zeros(3)
    with pytest.raises(ValueError, match="contiguous float32 CUDA tensor"):
        ops.batch_normalize_2d(x, [0, 1], True, 0.1, 1e-5)
    with pytest.raises(ValueError, match="contiguous float32 CUDA tensor"):
        ops.batch_normalize_adjoint([0, 1], x, x, v, v)
    with pytest.raises(ValueError, match="axes"):
        ops.batch_normalize_2d(x, [1, 2], True, 0.1, 1e-5)
    f, b = address("anode_gpu_batch_normalize_3d1_packed_f32"), address("anode_gpu_batch_normalize_adjoint_3d1_packed_f32")
    assert f(0, 3, 2, 1e-5, 0.1, *[None] * 8) == -2 and f(65536, 65536, 1, 1e-5, 0.1, *[None] * 8) == -2
    assert f(4, 3, 2, 1e-5, 0.1, *[None] * 8) == -1 and f(4, 3, 2, 1e-5, 0.1, 2, 16, 16, 16, None, None, None, None) == -6
    assert b(0, 3, 2, *[None] * 9) == -2 and b(4, 3, 2, *[None] * 9) == -1 and b(4, 3, 2, 2, 16, 16, 16, 16, 16, 16, None, None) == -6


def compare_with_float64(shape, seed=0):
    """Composition and adjoint of a large layer, reference computed on the device."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.randn(shape, device="cuda", generator=g).mul_(2.0).add_(0.5)
    dy = torch.randn(shape, device="cuda", generator=g)
    c, ax = shape[1], (0, 2, 3)
    am, av = torch.zeros(c, device="cuda"), torch.ones(c, device="cuda")
    y, mean, var, am, av = ops.batch_normalize_2d(x, [0, 1], True, 0.1, 1e-5, am, av)
    x64, bs, m = x.double(), (1, c, 1, 1), x.numel() // c
    wm, wv = x64.mean(ax), x64.var(ax, unbiased=False) + 1e-5
    for name, got, want in (("mean", mean, wm), ("var", var, wv), ("running mean", am, 0.1 * wm), ("running variance", av, 0.9 + 0.1 * wv),
                            ("y", y, (x64 - wm.view(bs)) / wv.sqrt().view(bs))):
        assert bool(((got.double() - want).abs() <= 1e-5 + 1e-4 * want.abs()).all()), (shape, name)
    dx, dmean, dvar = ops.batch_normalize_adjoint([0, 1], dy, x, mean, var)
    e, r, dy64 = x64 - mean.double().view(bs), var.double().rsqrt(), dy.double()
    wvar = (dy64 * e).sum(ax) * -0.5 * r / var.double()
    wmean = -r * dy64.sum(ax) - 2.0 * wvar * e.sum(ax) / m
    assert_sum_close(host(dvar), host(wvar), "dvar")
    assert_sum_close(host(dmean), host(wmean), "dmean")
    want = dy64 * r.view(bs) + (2.0 * wvar / m).view(bs) * e + (wmean / m).view(bs)
    assert bool(((dx.double() - want).abs() <= 1e-5 + 1e-4 * want.abs()).all()), (shape, "dx")


# one million floats to a channel and clusters for 148 SMs: the lines of normalized_apart
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(1337, 1, 28, 28), (1338, 1, 28, 28), (700, 3, 40, 40), (1338, 18, 28, 28), (1338, 19, 28, 28), (1100, 2, 31, 31)])
def test_large_layers_of_few_channels(shape):
    compare_with_float64(shape)


# rows that are loaded float by float, on both sides of eight blocks per SM and of 128 Ki floats to a channel
@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(3, 1024, 55, 55), (8, 600, 55, 55), (2, 2048, 55, 55), (6, 295, 55, 55), (6, 297, 55, 55), (44, 300, 55, 55)])
def test_scalar_rows_of_many_channels(shape):
    compare_with_float64(shape)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2657, 3, 56, 56), (2755, 3, 55, 55), (500, 64, 56, 56), (1000, 40, 28, 28), (40, 5, 28, 28)])
@pytest.mark.parametrize("value", [1.1, 0.7])
def test_the_sums_of_the_adjoint_are_no_less_exact_than_the_ops(shape, value):
    """Equal summands round the same way at every addition, so that a longer chain of additions shows."""
    c, ax, axes = shape[1], (0, 2, 3), [0, 1]
    x, dy = torch.full(shape, value, device="cuda"), torch.full(shape, 1.3 * value, device="cuda")
    zero, one = torch.zeros(c, device="cuda"), torch.ones(c, device="cuda")
    op_dvar, op_sum = torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
    ops.BatchNormalize2dBwdVarianceOp.apply(axes, dy, x, zero, one, op_dvar)
    ops.BatchNormalize2dBwdMeanOp.apply(axes, dy, one, op_sum)
    _, _, dvar = ops.batch_normalize_adjoint(axes, dy, x, zero, one)
    _, dmean, _ = ops.batch_normalize_adjoint(axes, dy, torch.zeros_like(x), zero, one)      # dmean is -sum(dy) alone
    want_dvar, want_sum = -0.5 * (dy.double() * x.double()).sum(ax), -dy.double().sum(ax)
    # (a sum and its product with -0.5 are rounded once each: 2^-23 beside the chain's own error)
    for got, op, want in ((dvar, op_dvar, want_dvar), (dmean, op_sum, want_sum)):
        err, err_op = (((t.double() - want) / want).abs().max().item() for t in (got, op))
        assert err <= err_op + 2.0 ** -22, (shape, value, err, err_op)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,kernel", [((2, 8, 7, 7), "register"), ((32, 64, 28, 28), "register"), ((9, 5, 55, 55), "register"),
                                          ((1024, 64, 7, 7), "stream"), ((2000, 20, 12, 12), "stream"), ((64, 8, 56, 56), "tiled")])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_the_mean_shows_an_infinity(shape, kernel, value):
    """As the ops' own: the mean and the running mean of a channel that holds an infinity are that infinity, those of one that
    holds both or a NaN are NaN; the variance and the output are NaN, and the other channels' results are what they are without."""
    assert ops.serving_kernel(shape, 0) == kernel
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x = torch.randn(shape, device="cuda", generator=g)
    c = shape[1]

    def run(x):
        return ops.batch_normalize_2d(x, [0, 1], True, 0.1, 1e-5, torch.zeros(c, device="cuda"), torch.ones(c, device="cuda"))
    clean = run(x)
    for places in (((0, 0, 0, 0),), ((-1, 0, -1, -1),), ((0, 0, 0, 1), (-1, 0, 0, 2))):
        p = x.clone()
        for q in places:
            p[q] = value
        p[0, 1, 0, 0], p[-1, 1, -1, -1] = float("inf"), float("-inf")
        y, mean, var, am, av = run(p)
        want = torch.full((), value)
        for t in (mean, am):
            assert torch.equal(t[:1].cpu().nan_to_num(7.0, 8.0, 9.0), want[None].nan_to_num(7.0, 8.0, 9.0)) and bool(t[1].isnan()), (places, t[:2])
        assert bool(var[:2].isnan().all() and av[:2].isnan().all() and y[:, :2].isnan().all())
        for got, ref in zip((y[:, 2:], mean[2:], var[2:], am[2:], av[2:]), (clean[0][:, 2:],) + tuple(t[2:] for t in clean[1:])):
            assert torch.equal(got, ref)


# forward passes that the streaming kernel serves, and large layers whose fused calls are other kernels' but whose composition is not
@pytest.mark.gpu
@pytest.mark.parametrize("shape,kernel", [((1024, 64, 7, 7), "stream"), ((512, 128, 7, 7), "stream"), ((2000, 20, 12, 12), "stream"),
                                          ((64, 8, 56, 56), "tiled"), ((64, 95, 55, 55), "tiled"), ((512, 64, 19, 19), "plain")])
def test_every_route_of_the_composition(shape, kernel):
    assert ops.serving_kernel(shape, 0) == kernel
    compare_with_float64(shape, seed=1)


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 512, 7, 7), (64, 8, 56, 56), (1024, 64, 7, 7), (1400, 2, 28, 28), (9, 60, 55, 55)])
def test_a_chain_of_overlapping_compositions(shape):
    """Each launch may begin before the one ahead of it on the stream has ended and reads what that one writes: the same results
    as with a synchronisation after every call, in a loop and as one captured graph."""
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    x, dy = torch.randn(shape, device="cuda", generator=g), torch.randn(shape, device="cuda", generator=g)
    am, av = torch.zeros(shape[1], device="cuda"), torch.ones(shape[1], device="cuda")

    def chain(after):
        am.zero_(), av.fill_(1.0)
        out, t = [], x
        for _ in range(3):
            y, mean, var, _, _ = ops.batch_normalize_2d(t, [0, 1], True, 0.1, 1e-5, am, av); after()
            y = ops.relu(y, inplace=True); after()
            dz = ops.PositiveClipBwdOp.apply(dy, y, torch.empty_like(y)); after()
            dx, dmean, dvar = ops.batch_normalize_adjoint([0, 1], dz, t, mean, var); after()
            out += [y, mean, var, dz, dx, dmean, dvar]
            t = dx
        return out + [am, av]
    want = [a.clone() for a in chain(torch.cuda.synchronize)]
    for _ in range(10):
        for i, (a, b) in enumerate(zip(chain(lambda: None), want)):
            assert torch.equal(a, b), i
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(lambda: None)
    for _ in range(3):
        graph.replay()
        for i, (a, b) in enumerate(zip(got, want)):
            assert torch.equal(a, b), i
