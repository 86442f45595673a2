"""Launches that overlap the kernel before them on the stream: every kernel of a chain reads what the one before wrote
(activations, statistics, running averages, parameters), so a load that is not behind the wait shows as a difference from
the same chain with a synchronisation after every call.  Also as one captured graph, and on a stream of its own."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(2, 512, 7, 7), (1, 53, 39, 25), (32, 64, 28, 28), (4, 16, 112, 112), (1411, 128, 7, 7), (64, 8, 56, 56),
          (1283, 244, 7, 7)]      # (the last one's forward and backward passes are cooperative launches of the band kernel)


def make(ops, shape):
    """Two layers, their buffers and the chain over them; the chain returns what it wrote."""
    c, axes = shape[1], [0, 1]
    layers = [ops.FusedBatchNormRelu(c), ops.FusedBatchNormRelu(c, relu=False)]
    g = torch.Generator(device="cuda")
    g.manual_seed(sum(shape))
    x = torch.randn(shape, device="cuda", generator=g)
    dy = torch.randn(shape, device="cuda", generator=g)
    t = [torch.zeros_like(x) for _ in range(8)]
    ws = ops.Workspace(*ops.dims_of(x), x.device)
    m, v = torch.zeros(c, device="cuda"), torch.ones(c, device="cuda")
    ops.FusedBatchNormRelu.forward(layers[0], x, out=t[0])          # makes the layers' workspaces
    ops.FusedBatchNormRelu.forward(layers[1], x, out=t[0])

    def reset():
        for layer in layers:
            layer.avg_mean.zero_(), layer.avg_var.fill_(1.0)
            if layer.gamma is not None:
                layer.gamma.fill_(1.0), layer.beta.zero_()

    def chain(after):
        a, b = layers
        for k in range(3):
            a.forward(x if k == 0 else t[3], out=t[0]); after()
            a.infer(t[0], out=t[1]); after()                         # running averages that the call before wrote
            b.forward(t[1], out=t[2]); after()
            b.infer(t[2], out=t[3]); after()
            b._x = t[1]
            b.backward(dy, out=t[4]); after()
            a._x = x if k == 0 else t[5]
            a.backward(t[4], out=t[6]); after()
            ops.BatchMean2dOp.apply(axes, t[6], m); after()
            ops.BatchVariance2dOp.apply(axes, 1e-5, t[6], m, v); after()
            ops.BatchNormalize2dOp.apply(axes, t[6], m, v, t[7]); after()
            ops.BatchNormalize2dActInferOp.apply(axes, t[7], m, v, t[5], a.dgamma, a.dbeta); after()
            ops.PositiveClipOp.apply(t[5], t[5]); after()
            ops.BatchNormalize2dAddActFusedOp.apply(axes, 1e-5, 0.1, t[5], t[3], t[3], a.mean, a.var, a.avg_mean, a.avg_var,
                                                    a.gamma, a.beta, workspace=ws); after()
            a.gamma.copy_(v); after()                                # another library's kernel in between
        return t[:8] + [m, v, a.mean, a.var, a.avg_mean, a.avg_var, a.dgamma, a.dbeta, b.avg_mean, b.avg_var]

    return reset, chain


@pytest.mark.parametrize("shape", SHAPES)
def test_a_chain_of_overlapping_launches(shape):
    from anode_b200 import ops
    reset, chain = make(ops, shape)
    reset()
    want = [a.clone() for a in chain(torch.cuda.synchronize)]
    assert all(torch.isfinite(a).all() for a in want)
    for _ in range(20):
        reset()
        got = chain(lambda: None)
        for i, (a, b) in enumerate(zip(got, want)):
            assert torch.equal(a, b), i
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        reset()
        got = [a.clone() for a in chain(lambda: None)]
    torch.cuda.current_stream().wait_stream(side)
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b), i
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = chain(lambda: None)
    for _ in range(5):
        reset()
        graph.replay()
        for i, (a, b) in enumerate(zip(got, want)):
            assert torch.equal(a, b), i
