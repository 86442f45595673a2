"""The work that users of this framework have it do, as cases that can be timed.

A case is one pass of one layer through the public entry points of `anode_b200.ops`: a training step
(forward and backward) of a batch-norm + ReLU layer, the same with the activation and write options of the
op constructors, the residual-block epilogue in both directions, the evaluation-mode pass, the op-by-op
composition that the graph front end builds, and the step on host tensors.  Every tensor is f32, the only
type of this path.

Kinds
  layer      FusedBatchNormRelu.forward, .backward
  ops        BatchNormalize2dFusedOp, BatchNormalize2dBwdFusedOp with a leaky ReLU, dx assigned or accumulated
  residual   BatchNormalize2dAddActFusedOp.apply, .adjoint
  infer      FusedBatchNormRelu.infer
  composed   batch_normalize_2d, relu in place, PositiveClipBwdOp, batch_normalize_adjoint
  host       FusedBatchNormRelu.step_from_host on page-locked tensors

Ranges: 2e4 to 1.6e9 elements for training steps and inference (host tensors 1e5 to 1.5e7), 3 to 2048
channels, spatial sides of 4 to 160 in two dimensions and 4 to 128 in three, batches of 1 to 4096.
"""
import torch

from anode_b200 import ops

EPSILON, AVG_RATE = 1e-5, 0.1


def case_of(kind, n, c, d, h, w, **options):
    case = dict(kind=kind, n=n, c=c, d=d, h=h, w=w, dist="normal", affine=True, relu=True, slope=0.0, accumulate=False)
    case.update(options)
    return case


def listed():
    return [
        # a late layer at a batch of two: nothing but latency, launches and the host path
        case_of("layer", 2, 512, 0, 7, 7, name="step_smallest"),
        # the correctness configuration: a small layer at an ordinary batch
        case_of("layer", 32, 64, 0, 28, 28, name="step_small"),
        # the ResNet stem at a batch of 256
        case_of("layer", 256, 64, 0, 112, 112, name="step_stem"),
        # a U-Net volume: four samples, rows of two million elements
        case_of("layer", 4, 32, 128, 128, 128, name="step_volume"),
        # wide channels, 7 x 7 rows, heavy tails: the last stage of a ResNet at a batch of 1024
        case_of("layer", 1024, 2048, 0, 7, 7, dist="student3", name="step_wide"),
        # the global batch of the benchmark's main configuration on one GPU: the largest call
        case_of("layer", 2048, 256, 0, 56, 56, name="step_largest"),
        # sizes that divide by nothing (odd rows, odd channel count), with a leaky ReLU
        case_of("ops", 64, 95, 0, 55, 55, slope=0.1, name="ragged_leaky"),
        # the end of a residual block in the third and in the first stage of a ResNet
        case_of("residual", 256, 1024, 0, 14, 14, name="residual_mid"),
        case_of("residual", 256, 256, 0, 56, 56, name="residual_long"),
        # evaluation at a serving batch
        case_of("infer", 8, 256, 0, 28, 28, name="infer_serving"),
        # the graph front end's own composition, op by op
        case_of("composed", 64, 128, 0, 28, 28, name="composed_ops"),
        # a layer whose tensors live in host memory
        case_of("host", 64, 64, 0, 56, 56, name="host_step"),
    ]


SIDES_2D = (7, 8, 14, 16, 28, 32, 56, 64, 112, 128)
SIDES_3D = (8, 16, 24, 32, 48, 64, 96, 128)
CHANNELS = (16, 32, 64, 128, 256, 512, 1024, 2048)
#: kind -> (share of the draws, smallest and largest element count)
DRAWN = {"layer": (0.46, 2e4, 4e8), "ops": (0.12, 2e4, 2e8), "residual": (0.14, 2e4, 4e8), "infer": (0.12, 2e4, 4e8),
         "composed": (0.10, 2e4, 5e7), "host": (0.06, 1e5, 1.5e7)}


def log_uniform(rng, low, high):
    return low * (high / low) ** rng.random()


def draw(rng):
    kind = rng.choices(list(DRAWN), [v[0] for v in DRAWN.values()])[0]
    elements = log_uniform(rng, *DRAWN[kind][1:])
    common = rng.random() < 0.6
    if rng.random() < 0.85:
        d, (h, w) = 0, [rng.choice(SIDES_2D)] * 2 if common else [round(log_uniform(rng, 4, 160)) for _ in range(2)]
    else:
        d, h, w = [rng.choice(SIDES_3D)] * 3 if common else [round(log_uniform(rng, 4, 64)) for _ in range(3)]
    row = max(1, d) * h * w
    c = rng.choice(CHANNELS) if rng.random() < 0.6 else round(log_uniform(rng, 3, 2048))
    c = max(3, min(c, int(elements // row)))
    n = max(1, min(4096, round(elements / (row * c))))
    case = case_of(kind, n, c, d, h, w, dist="student3" if rng.random() < 0.15 else "normal",
                   affine=rng.random() < 0.85, relu=kind not in ("layer", "infer") or rng.random() < 0.9)
    if kind == "ops":
        case.update(slope=rng.choice((0.01, 0.1, 0.2)), accumulate=rng.random() < 0.3)
    return case


def shape_of(case):
    return (case["n"], case["c"]) + ((case["d"],) if case["d"] else ()) + (case["h"], case["w"])


def activations(case, g):
    """The output of a convolution: N(mean of the channel, 2), or 4 * Student-t with three degrees of freedom.  The
    values lie on a grid of 1/32 (about the resolution of bf16 at their size), so that rounding in the statistics
    does not decide on which side of the ReLU's threshold an element falls."""
    shape, c = shape_of(case), case["c"]
    x = torch.randn(shape, device="cuda", generator=g)
    if case["dist"] == "student3":
        chi = torch.zeros_like(x)
        for _ in range(3):
            z = torch.randn(shape, device="cuda", generator=g)
            chi.addcmul_(z, z)
            del z
        x.mul_(chi.div_(3.0).rsqrt_()).mul_(4.0)
        del chi
    else:
        mean = torch.rand(c, device="cuda", generator=g) * 2.0 - 1.0
        x.mul_(2.0).add_(mean.view((1, c) + (1,) * (len(shape) - 2)))
    return x.mul_(32.0).round_().div_(32.0)


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    shape, c, kind = shape_of(case), case["c"], case["kind"]
    x = activations(case, g)
    s = dict(case=case, axes=list(range(len(shape) - 2)), x=x)
    layer = s["layer"] = ops.FusedBatchNormRelu(c, EPSILON, AVG_RATE, affine=case["affine"], relu=case["relu"])
    if case["affine"]:
        layer.gamma.copy_(torch.rand(c, device="cuda", generator=g) + 0.5)
        layer.beta.copy_(torch.rand(c, device="cuda", generator=g) * 0.2 - 0.1)
    if kind == "infer":
        layer.avg_mean.copy_(torch.rand(c, device="cuda", generator=g) * 2.0 - 1.0)
        layer.avg_var.copy_(torch.rand(c, device="cuda", generator=g) * 4.0 + 2.0)
        s["y"] = torch.empty_like(x)
        return s
    s["dy"] = torch.randn(shape, device="cuda", generator=g)
    if kind == "composed":
        s["dz"] = torch.empty_like(x)
        return s
    if kind == "residual":      # the shortcut is a ReLU's output, too (on a coarser grid, for the same reason as x)
        s["shortcut"] = torch.randn(shape, device="cuda", generator=g).mul_(8.0).round_().div_(8.0).clamp_min_(0.0)
        s["dshortcut"] = torch.empty_like(x)
    if kind == "host":
        for k in ("x", "dy"):
            s[k] = s[k].cpu().pin_memory()
        for k in ("y", "dx"):
            s[k] = torch.zeros(shape).pin_memory()
        return s
    s["y"], s["dx"] = torch.empty_like(x), torch.zeros_like(x)
    if kind in ("ops", "residual"):
        s["workspace"] = ops.Workspace(*ops.dims_of(x), x.device)
    return s


def run(s):
    return RUN[s["case"]["kind"]](s)


def statistics_of(layer):
    return dict(mean=layer.mean, var=layer.var, avg_mean=layer.avg_mean, avg_var=layer.avg_var, dgamma=layer.dgamma, dbeta=layer.dbeta)


def run_layer(s):
    layer = s["layer"]
    y = layer.forward(s["x"], out=s["y"])
    dx = layer.backward(s["dy"], out=s["dx"])
    return dict(statistics_of(layer), y=y, dx=dx)


def run_ops(s):
    layer, case = s["layer"], s["case"]
    y = ops.BatchNormalize2dFusedOp.apply(
        s["axes"], EPSILON, AVG_RATE, s["x"], s["y"], layer.mean, layer.var, layer.avg_mean, layer.avg_var, layer.gamma,
        layer.beta, workspace=s["workspace"], neg_slope=case["slope"])
    dx = ops.BatchNormalize2dBwdFusedOp.apply(
        s["axes"], s["dy"], s["x"], layer.mean, layer.var, s["dx"], layer.gamma, layer.beta, layer.dgamma, layer.dbeta,
        cap=ops.WriteCap.Accumulate if case["accumulate"] else ops.WriteCap.Assign, workspace=s["workspace"],
        neg_slope=case["slope"])
    return dict(statistics_of(layer), y=y, dx=dx)


def run_residual(s):
    layer = s["layer"]
    op = ops.BatchNormalize2dAddActFusedOp
    y = op.apply(s["axes"], EPSILON, AVG_RATE, s["x"], s["shortcut"], s["y"], layer.mean, layer.var, layer.avg_mean,
                 layer.avg_var, layer.gamma, layer.beta, workspace=s["workspace"])
    dx, dshortcut = op.adjoint(s["axes"], s["dy"], s["x"], y, layer.mean, layer.var, s["dx"], s["dshortcut"], layer.gamma,
                               layer.beta, layer.dgamma, layer.dbeta, workspace=s["workspace"])
    return dict(statistics_of(layer), y=y, dx=dx, dshortcut=dshortcut)


def run_infer(s):
    return s["layer"].infer(s["x"], out=s["y"])


def run_composed(s):
    layer = s["layer"]
    y, mean, var, avg_mean, avg_var = ops.batch_normalize_2d(s["x"], s["axes"], True, AVG_RATE, EPSILON, layer.avg_mean, layer.avg_var)
    y = ops.relu(y, inplace=True)
    dz = ops.PositiveClipBwdOp.apply(s["dy"], y, s["dz"])
    dx, dmean, dvar = ops.batch_normalize_adjoint(s["axes"], dz, s["x"], mean, var)
    return dict(y=y, mean=mean, var=var, avg_mean=avg_mean, avg_var=avg_var, dz=dz, dx=dx, dmean=dmean, dvar=dvar)


def run_host(s):
    layer = s["layer"]
    layer.step_from_host(s["x"], s["dy"], s["y"], s["dx"])
    return dict(statistics_of(layer), y=s["y"], dx=s["dx"])


RUN = dict(layer=run_layer, ops=run_ops, residual=run_residual, infer=run_infer, composed=run_composed, host=run_host)

#: passes over a tensor that a pass of each kind cannot do without (f32: 4 bytes each), and operations per element
TENSORS = {"layer": 5,          # x, y; x, dy, dx
           "ops": 5,
           "residual": 8,       # x, shortcut, y; x, dy, y, dx, dshortcut
           "infer": 2,          # x, y
           "composed": 10,      # x, y; y, y; dy, y, dz; x, dz, dx
           "host": 4}           # x, dy in, y, dx out over the link
FLOPS = {"layer": 14, "ops": 14, "residual": 16, "infer": 3, "composed": 14, "host": 14}


def work(case):
    elements = 1
    for v in shape_of(case):
        elements *= v
    tensors = TENSORS[case["kind"]] + (1 if case["accumulate"] else 0)
    return {"bytes": 4.0 * (tensors * elements + 10 * case["c"]), "flops": float(FLOPS[case["kind"]] * elements)}


def tolerance(case):
    # 32-bit sums and elementwise arithmetic; the largest differences are those of channel sums that cancel
    return {"rel": 2e-5, "max": 1e-3}
