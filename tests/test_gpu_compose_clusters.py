"""The adjoint of the composition (and its forward pass over scalar rows) where the number of blocks per channel changes, and at
channels that are just held by a block's threads, by several vectors each, or not: against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# clusters of eight, four, two and one, on both sides of each line, rows that are loaded by vectors and float by float
CLUSTERS = [(n, c) + hw for c in (37, 38, 74, 75, 148, 149, 300) for n, hw in ((600, (8, 8)), (301, (7, 7)))]
# one block: threads of 64 floats and more have two; channels that two blocks hold; up to four vectors held per thread, blocks of all sizes
EDGES = [(2048, 150, 4, 4), (2047, 150, 4, 4), (669, 150, 7, 7), (668, 150, 7, 7), (1024, 150, 4, 4), (1025, 150, 4, 4), (513, 150, 4, 4),
         (9, 2048, 5, 5), (16, 2048, 7, 7), (20, 2048, 8, 8), (128, 700, 8, 8), (129, 700, 8, 8), (1, 2500, 1, 3)]
# channels that a cluster of eight or four holds: on both sides of the lines between it and smaller ones by the number of blocks; and channels
# whose second walk is kept within reach of L2
HELD = [(64, c, 28, 28) for c in (35, 36, 70, 71, 75, 88, 89, 150, 185, 186)] + [(37, 149, 28, 28), (24, 310, 28, 28), (14, 300, 40, 55)]
WINDOWS = [(127, 128, 32, 32), (256, 150, 28, 28), (33, 186, 55, 55)]


@pytest.mark.parametrize("shape", CLUSTERS + EDGES + HELD + WINDOWS)
def test_adjoint_and_composition(shape):
    from anode_b200 import ops
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(shape))
    c, m = shape[1], shape[0] * shape[2] * shape[3]
    x = torch.randn(shape, device="cuda", generator=g) * 2 + 1
    dy = torch.randn(shape, device="cuda", generator=g)
    mean, var = torch.randn(c, device="cuda", generator=g), torch.rand(c, device="cuda", generator=g) + 0.5
    v = lambda t: t.double().view(1, -1, 1, 1)
    e, r = x.double() - v(mean), 1 / var.double().sqrt()
    dvar = (dy.double() * e).sum((0, 2, 3)) * -0.5 * r / var.double()
    dmean = -r * dy.double().sum((0, 2, 3)) - 2 * dvar * e.sum((0, 2, 3)) / m
    dx = dy.double() * v(r) + v(2 * dvar / m) * e + v(dmean / m)
    batch_mean, batch_var = x.double().mean((0, 2, 3)), x.double().var((0, 2, 3), unbiased=False) + 1e-5
    got = ops.batch_normalize_adjoint([0, 1], dy, x, mean, var)
    ops.set_kernel("plain")                     # the composition's own kernel
    try:
        fwd = ops.batch_normalize_2d(x, [0, 1], True, 0.1, 1e-5)
    finally:
        ops.set_kernel("auto")
    for a, w, what in ((got[0], dx, "dx"), (got[1], dmean, "dmean"), (got[2], dvar, "dvar"), (fwd[1], batch_mean, "mean"), (fwd[2], batch_var, "var"),
                       (fwd[0], (x.double() - v(batch_mean)) / v(batch_var.sqrt()), "y")):
        # 1e-4 of the value and 1e-5, channel sums also 1e-4 of their root mean square (tests/util.py)
        atol = 1e-5 + (1e-4 * float(w.square().mean().sqrt()) if what in ("dmean", "dvar") else 0.0)
        assert not ((a.double() - w).abs() > atol + 1e-4 * w.abs()).any(), (shape, what)
