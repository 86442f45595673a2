"""The native call module (csrc/bn_py.cpp) refuses what it cannot take with a Python error, on any machine: nothing of a
refused call reaches CUDA, and no C++ exception leaves the module."""
import numpy as np
import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from anode_b200 import _lib, build, ops


class Scratch:
    """Stands in for ops.Workspace, whose constructor needs a device."""
    def __init__(self):
        self.buf, self.bytes = torch.empty(256, dtype=torch.uint8), 256


def calls(x, v):
    """Every op that goes through the module, on activations x and per-channel vectors v."""
    ax, f, b, r = [0, 1], ops.BatchNormalize2dFusedOp.apply, ops.BatchNormalize2dBwdFusedOp.apply, ops.BatchNormalize2dAddActFusedOp
    ws = Scratch()
    return {
        "fwd": lambda: f(ax, 1e-5, 0.1, x, x, v, v, workspace=ws),
        "fwd leaky": lambda: f(ax, 1e-5, 0.1, x, x, v, v, workspace=ws, neg_slope=0.1),
        "bwd": lambda: b(ax, x, x, v, v, x, workspace=ws),
        "residual fwd": lambda: r.apply(ax, 1e-5, 0.1, x, x, x, v, v, workspace=ws),
        "residual bwd": lambda: r.adjoint(ax, x, x, x, v, v, x, workspace=ws),
        "infer": lambda: ops.BatchNormalize2dActInferOp.apply(ax, x, v, v, x),
        "mean": lambda: ops.BatchMean2dOp.apply(ax, x, v),
        "mean bwd": lambda: ops.BatchMean2dBwdOp.apply(ax, v, x, x),
        "var": lambda: ops.BatchVariance2dOp.apply(ax, 1e-5, x, v, v),
        "var bwd": lambda: ops.BatchVariance2dBwdOp.apply(ax, v, x, v, x),
        "var bwd mean": lambda: ops.BatchVariance2dBwdMeanOp.apply(ax, v, x, v, v),
        "norm": lambda: ops.BatchNormalize2dOp.apply(ax, x, v, v, x),
        "norm bwd": lambda: ops.BatchNormalize2dBwdOp.apply(ax, x, v, x),
        "norm bwd var": lambda: ops.BatchNormalize2dBwdVarianceOp.apply(ax, x, x, v, v, v),
        "clip": lambda: ops.PositiveClipOp.apply(x, x),
        "clip bwd": lambda: ops.PositiveClipBwdOp.apply(x, x, x),
        "join": lambda: ops.FlatJoinOp.apply(x, x, x),
    }


NAMES = sorted(calls(None, None))


@pytest.mark.parametrize("name", NAMES)
def test_host_tensors_are_refused_before_anything_is_asked_of_cuda(name):
    with pytest.raises(ValueError, match="contiguous float32 CUDA tensor"):
        calls(torch.zeros(2, 3, 4, 4), torch.zeros(3))[name]()


@pytest.mark.parametrize("name", NAMES)
def test_tensors_without_storage_raise(name):
    with FakeTensorMode():
        x, v = torch.empty(5, 2, 3, 4, 4, device="cuda"), torch.empty(5, 3, device="cuda")

        def one(x, v):
            return calls(x, v)[name]()
        with pytest.raises(RuntimeError):
            torch.func.vmap(one)(x, v)


@pytest.mark.skipif(torch.cuda.is_available(), reason="needs a machine without a driver")
@pytest.mark.filterwarnings("ignore:Accessing the data pointer of FakeTensor")
def test_no_driver_is_an_error_not_an_abort():
    with FakeTensorMode():
        x, v = torch.empty(2, 3, 4, 4, device="cuda"), torch.empty(3, device="cuda")
    with pytest.raises(RuntimeError):
        ops.BatchNormalize2dActInferOp.apply([0, 1], x, v, v, x)      # asks for the current stream


def test_the_form_of_a_call_never_depends_on_its_arguments():
    """Values that once chose between the C calls' forms are refused like any other wrong ones."""
    x, v = torch.zeros(2, 3, 4, 4), torch.zeros(3)
    with pytest.raises(TypeError):
        ops.BatchVariance2dOp.apply([0, 1], None, x, v, v)             # no epsilon
    with pytest.raises(TypeError):
        ops.BatchMean2dOp.apply(False, x, v)                          # no axes: not the flat form
    with pytest.raises(TypeError):
        ops.BatchNormalize2dBwdOp.apply(False, x, v, x)


@pytest.mark.parametrize("call", [lambda x, v: ops.BatchMean2dOp.apply([0, 1], x, None), lambda x, v: ops.PositiveClipOp.apply(None, x),
                                  lambda x, v: ops.BatchNormalize2dOp.apply([0, 1], x, None, v, x)])
def test_the_references_entry_points_take_no_missing_array(call):
    """They have no status to answer with: a missing array would be read."""
    with pytest.raises((ValueError, AttributeError)):
        call(torch.zeros(2, 3, 4, 4), torch.zeros(3))


def entries(axes, **kw):
    """One op of each kind with these axes, on host tensors, with a workspace where one is taken."""
    x, v = torch.zeros(2, 3, 4, 4), torch.zeros(3)
    fused = dict(kw, workspace=Scratch())
    return [lambda: ops.BatchMean2dOp.apply(axes(), x, v, **kw), lambda: ops.BatchVariance2dOp.apply(axes(), 1e-5, x, v, v, **kw),
            lambda: ops.BatchNormalize2dActInferOp.apply(axes(), x, v, v, x, **kw),
            lambda: ops.BatchNormalize2dFusedOp.apply(axes(), 1e-5, 0.1, x, x, v, v, **fused),
            lambda: ops.BatchNormalize2dBwdFusedOp.apply(axes(), x, x, v, v, x, **fused),
            lambda: ops.BatchNormalize2dAddActFusedOp.apply(axes(), 1e-5, 0.1, x, x, x, v, v, **fused),
            lambda: ops.BatchNormalize2dAddActFusedOp.adjoint(axes(), x, x, x, v, v, x, **fused)]


@pytest.mark.parametrize("axes", [lambda: [0, 1], lambda: (0, 1), lambda: range(2), lambda: iter([0, 1]), lambda: {0: 0, 1: 0},
                                  lambda: np.arange(2), lambda: torch.arange(2), lambda: [0.0, 1.0], lambda: None],
                         ids=["list", "tuple", "range", "iterator", "keys", "numpy", "torch", "floats", "unchecked"])
def test_axes_are_any_iterable_of_the_positions(axes):
    for call in entries(axes):
        with pytest.raises(ValueError, match="contiguous float32 CUDA tensor"):      # the axes were taken
            call()


@pytest.mark.parametrize("axes", [[1, 0], [0], [0, 1, 2], [], "ab"])
def test_other_axes_are_refused(axes):
    for call in entries(lambda: axes):
        with pytest.raises(ValueError, match="axes must be"):
            call()
    x, v = torch.zeros(2, 3, 4, 4), torch.zeros(3)
    with pytest.raises(ValueError, match="axes must be"):          # and before a workspace is made
        ops.BatchNormalize2dFusedOp.apply(axes, 1e-5, 0.1, x, x, v, v)
    with pytest.raises(TypeError):
        ops.BatchMean2dOp.apply(7, x, v)


def test_a_launch_hint_is_one():
    x = torch.zeros(2, 3, 4, 4)
    for call in entries(lambda: [0, 1], cfg="1024") + [lambda: ops.PositiveClipOp.apply(x, x, cfg=1024)]:
        with pytest.raises(TypeError):
            call()
    for call in entries(lambda: [0, 1], cfg=ops.KernelConfig(256, 148)):
        with pytest.raises(ValueError, match="contiguous float32 CUDA tensor"):
            call()


def test_the_residual_epilogue_has_a_slope():
    x, v = torch.zeros(2, 3, 4, 4), torch.zeros(3)
    with pytest.raises(TypeError):
        ops.BatchNormalize2dAddActFusedOp.apply([0, 1], 1e-5, 0.1, x, x, x, v, v, neg_slope=None, workspace=Scratch())
    with pytest.raises(TypeError):
        ops.BatchNormalize2dAddActFusedOp.adjoint([0, 1], x, x, x, v, v, x, neg_slope=None, workspace=Scratch())


def test_the_module_is_bound_to_this_interpreter_and_torch(tmp_path, monkeypatch):
    assert _lib.native().built_for == build.native_built_for()
    assert build.native_is_current(build.NATIVE, build.NATIVE_SOURCE, build.native_built_for())
    assert not build.native_is_current(build.NATIVE, build.NATIVE_SOURCE, "built for cpython-311, torch 2.0")     # built again
    assert not build.native_is_current(str(tmp_path / "missing.so"), build.NATIVE_SOURCE, build.native_built_for())
    monkeypatch.setattr(build, "native_built_for", lambda: "built for cpython-311, torch 2.0")
    monkeypatch.setattr(_lib, "_native", None)
    with pytest.raises(ImportError, match="built for cpython-311"):        # and not used in the meantime
        _lib.native()
