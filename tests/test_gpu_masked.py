"""The streaming kernel's masked form: runs of channels that begin anywhere in a 16-byte vector.  Its index arithmetic on the CPU
(every element of the tensor in one lane of one thread, each lane folded into the channel it belongs to, no access outside the
tensor), and its results where the splits have remainders: strides of every remainder by four, a tensor that ends inside a vector,
one sample and one channel, a last unit of fewer channels, more groups than samples, clusters of sixteen."""
import ctypes

import numpy as np
import pytest
import torch

from tests.test_gpu_fused import run_fused
from tests.test_gpu_random_shapes import run_add_act
from tests.test_gpu_tiled_forms import outputs_over_inputs
from tests.util import check_layer_own_mask, make_inputs

SHAPES = [(1411, 127, 7, 7), (301, 3, 5, 5), (4099, 5, 1, 5), (7, 3, 3, 3), (1, 3, 1, 5), (1, 1, 1, 7), (2, 1, 1, 9), (333, 23, 11, 11),
          (64, 4, 19, 19), (512, 64, 19, 19), (45, 33, 1, 237), (1283, 21, 1, 94), (4100, 3, 1, 77), (2000, 5, 1, 6), (63, 130, 1, 253),
          (3, 1, 1, 250), (17, 91, 13, 13), (2571, 13, 1, 75)]


def masked_geometry(shape, direction, residual):
    from anode_b200 import _lib
    n, c, d0 = shape[0], shape[1], shape[2] * shape[3]
    out = (ctypes.c_uint32 * 7)()
    assert _lib.load().anode_gpu_batch_norm_stream_masked_geometry(d0, c, n, direction, residual, out) == 0
    return dict(zip(["applies", "cb", "units", "cluster", "rows", "groups", "threads"], list(out)))


@pytest.mark.parametrize("shape", [s for s in SHAPES if s[0] * s[1] * s[2] * s[3] < 3e5])
@pytest.mark.parametrize("direction,residual", [(0, 0), (1, 0), (1, 1)])
def test_every_element_has_one_lane(shape, direction, residual):
    n, c, d0 = shape[0], shape[1], shape[2] * shape[3]
    g = masked_geometry(shape, direction, residual)
    assert g["applies"] == 1 and g["cb"] <= 128 and g["cb"] * g["cluster"] <= 1024 and g["units"] == -(-c // g["cb"])
    assert g["cluster"] in (1, 2, 4, 8, 16) and g["cluster"] * g["rows"] >= n and 1 <= g["groups"] <= g["rows"]
    rs, total = c * d0, n * c * d0
    assert g["rows"] <= g["groups"] or g["groups"] * rs % 4 == 0      # a thread of several samples: all lie alike
    seen, folded = np.zeros(total, np.int32), np.zeros((c, total), bool) if c * total < 3e7 else None
    for u in range(g["units"]):
        c0 = u * g["cb"]
        cw = min(c - c0, g["cb"])
        run, vectors = cw * d0, (cw * d0 + 6) // 4
        assert g["groups"] * vectors <= g["threads"] <= 256
        for rank in range(g["cluster"]):
            n0 = rank * g["rows"]
            rows = min(max(n - n0, 0), g["rows"])
            lanes = {}                                               # (group, vector) -> channel of the first part, first lane of the second, elements
            for grp in range(g["groups"]):
                for v in range(vectors):
                    start = (n0 + grp) * rs + c0 * d0
                    mis = start % 4
                    lo, hi = (mis if v == 0 else 0), max(0, min(4, run + mis - 4 * v))
                    if grp >= rows or lo >= hi:
                        continue
                    first = (4 * v + lo - mis) // d0
                    limit = (first + 1) * d0 + mis - 4 * v
                    part = {}
                    for k in range(grp, rows, g["groups"]):
                        at = (n0 + k) * rs + c0 * d0 - mis + 4 * v
                        assert at % 4 == 0 and ((n0 + k) * rs + c0 * d0) % 4 == mis
                        for e in range(lo, hi):
                            seen[at + e] += 1
                            part.setdefault(int(e >= limit), []).append(at + e)
                    lanes[grp, v] = part
            if folded is None:
                continue
            for ci in range(cw):                                     # the fold of channel ci, as the kernel walks it
                f0 = ci * d0
                for i in range((d0 + 6) // 4 * g["groups"]):
                    gi = i // ((d0 + 6) // 4)
                    m = ((n0 + gi) * rs + c0 * d0) % 4
                    vi = (f0 + m) // 4 + i - gi * ((d0 + 6) // 4)
                    if 4 * vi >= f0 + d0 + m:
                        continue
                    for at in lanes.get((gi, vi), {}).get(int(ci > 0 and 4 * vi < f0 + m), []):
                        assert not folded[c0 + ci, at]
                        folded[c0 + ci, at] = True
    assert (seen == 1).all()
    if folded is not None:
        channel = np.arange(total) // d0 % c
        assert (folded == (channel[None] == np.arange(c)[:, None])).all()


def test_only_rows_without_an_aligned_run():
    for shape in ((1024, 2048, 7, 7), (64, 16, 7, 7), (2, 512, 7, 7), (9, 3, 1, 3), (9, 4, 1, 1), (5, 3, 1, 1100)):
        assert masked_geometry(shape, 0, 0)["applies"] == 0, shape
    assert masked_geometry((8, 3, 1, 253), 0, 0)["applies"] == 1


@pytest.fixture
def stream():
    from anode_b200 import ops
    ops.set_kernel("stream")
    yield ops
    ops.set_kernel("auto")


@pytest.mark.gpu
@pytest.mark.parametrize("shape", SHAPES)
def test_layers(stream, shape):
    ops = stream
    assert [ops.serving_kernel(shape, d, residual=r) for r in (False, True) for d in (0, 1)] == ["stream"] * 4
    d = make_inputs(shape, seed=sum(shape), loc=3.0, scale=2.0)
    got, ws = run_fused(ops, d)
    assert ops.last_kernel() == "stream"
    check_layer_own_mask(d, got, "%r " % (shape,))
    again, _ = run_fused(ops, d, ws=ws)
    for k in ("y", "dx", "mean", "var"):
        assert np.array_equal(again[k], got[k]), (shape, k)
    res = np.random.default_rng(5).standard_normal(shape).astype(np.float32)
    for slope in (0.0, 0.1):
        got = run_add_act(ops, d, res, slope)
        check_layer_own_mask(d, got, "%r slope %g " % (shape, slope), residual=res, slope=slope)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["dres is dy", "dres is y", "dres is x", "no dres", "dx is dy", "dx is x", "accumulate"])
def test_outputs_over_inputs(form):
    from anode_b200 import ops
    outputs_over_inputs(ops, (1411, 13, 7, 7), form, "stream")


@pytest.mark.gpu
def test_a_channel_with_a_nan_or_an_infinity_leaves_its_neighbours_alone(stream):
    shape = (700, 11, 5, 5)
    d = make_inputs(shape, seed=9, loc=1.0, scale=2.0)
    want, _ = run_fused(stream, d)
    d["x"][3, 4, 0, 0], d["x"][699, 4, 4, 4], d["x"][5, 8, 4, 4] = np.nan, np.inf, -np.inf
    got, _ = run_fused(stream, d)
    for k in ("mean", "var", "dgamma", "dbeta"):
        assert not np.isfinite(got[k][[4, 8]]).any() or k == "dbeta"
    rest = [i for i in range(11) if i not in (4, 8)]
    for k in ("y", "dx"):
        assert np.array_equal(got[k][:, rest], want[k][:, rest]), k


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(4096, 23, 7, 7), (512, 64, 19, 19)])
def test_it_serves_what_the_plain_kernel_is_named_for(shape):
    from anode_b200 import ops
    assert [ops.serving_kernel(shape, d) for d in (0, 1)] == ["plain"] * 2
    d = make_inputs(shape, seed=1, loc=1.0, scale=2.0)
    got, _ = run_fused(ops, d)
    assert ops.last_kernel() == "stream"
    check_layer_own_mask(d, got, "%r " % (shape,))


@pytest.mark.gpu
@pytest.mark.parametrize("shape,named,launched", [
    ((1384, 111, 1, 18), ["register"] * 4, ["stream"] * 4), ((67, 706, 1, 37), ["register"] * 4, ["register"] * 3 + ["stream"]),
    ((16, 2017, 1, 151), ["register"] * 4, ["register"] * 4), ((604, 18, 13, 17), ["tiled"] * 4, ["stream"] * 4),
    ((4294, 15, 1, 254), ["tiled"] * 4, ["tiled"] * 4), ((1841, 15, 1, 165), ["tiled"] * 3 + ["plain"], ["stream"] * 4)])
def test_where_it_is_launched(shape, named, launched):
    from anode_b200 import ops
    assert [ops.serving_kernel(shape, d, residual=r) for r in (False, True) for d in (0, 1)] == named
    d = make_inputs(shape, seed=sum(shape), loc=1.0, scale=2.0)
    x, dy = torch.from_numpy(d["x"]).cuda(), torch.from_numpy(d["dy"]).cuda()
    c, got, op = shape[1], [], ops.BatchNormalize2dAddActFusedOp
    z = lambda: torch.zeros(c, device="cuda")
    mean, var, rm, rv, dg, db, y, dx, dr = z(), z(), z(), z(), z(), z(), torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    ws = ops.Workspace(*ops.dims_of(x), x.device)
    for call in (lambda: ops.BatchNormalize2dFusedOp.apply([0, 1], 1e-5, 0.1, x, y, mean, var, rm, rv, None, None, workspace=ws, neg_slope=0.0),
                 lambda: ops.BatchNormalize2dBwdFusedOp.apply([0, 1], dy, x, mean, var, dx, None, None, dg, db, workspace=ws, neg_slope=0.0),
                 lambda: op.apply([0, 1], 1e-5, 0.1, x, dy, y, mean, var, rm, rv, None, None, 0.0, ws),
                 lambda: op.adjoint([0, 1], dy, x, y, mean, var, dx, dr, None, None, dg, db, 0.0, workspace=ws)):
        call()
        got.append(ops.last_kernel())
    assert got == launched and ws.status() == 0
    run, _ = run_fused(ops, d)
    check_layer_own_mask(d, run, "%r " % (shape,))
