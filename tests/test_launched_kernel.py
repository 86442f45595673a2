"""Which kernel a call launches depends on the call alone: not on the shapes that its thread saw before, whose plans lay at the same
place of the thread's table.  Shapes that the streaming kernel and the kernel for long rows both take; on the GPU the launched kernel
and the outputs' bits, too."""
import threading

import numpy as np
import pytest

from anode_b200 import ops
from tests.test_gpu_fused import run_fused
from tests.util import check_layer_own_mask, make_inputs

# (call, direction, residual epilogue, shapes seen before it, in this order)
CALLS = [((169, 32, 1, 254), 1, True, [(2062, 23, 1, 49)]), ((207, 54, 1, 262), 1, False, [(1024, 95, 11, 11)]),
         ((156, 32, 1, 262), 1, True, [(1024, 95, 11, 11)]), ((4096, 23, 7, 7), 0, False, [(169, 32, 1, 254)]),
         ((947, 13, 1, 350), 0, False, [(604, 18, 13, 17)])]


def in_a_fresh_thread(f):
    got = []
    t = threading.Thread(target=lambda: got.append(f()))
    t.start()
    t.join()
    return got[0]


def asked(shape, direction, residual, before):
    for b in before:
        ops.launched_kernel(b, direction, residual)
    return ops.launched_kernel(shape, direction, residual)


@pytest.mark.parametrize("shape,direction,residual,before", CALLS)
def test_does_not_depend_on_calls_before(shape, direction, residual, before):
    fresh = in_a_fresh_thread(lambda: asked(shape, direction, residual, []))
    assert in_a_fresh_thread(lambda: asked(shape, direction, residual, before)) == fresh


def test_random_calls_in_any_order():
    rng = np.random.default_rng(3)
    shapes = [(int(rng.integers(20, 400)), int(rng.integers(8, 400)), 1, int(rng.integers(126, 256)) * 2) for _ in range(150)]
    fill = [(int(n), int(c), 1, int(d)) for n, c, d in zip(rng.integers(500, 4000, 400), rng.integers(5, 200, 400), rng.integers(9, 120, 400))]
    fresh = [in_a_fresh_thread(lambda s=s: [asked(s, d, r, []) for d in (0, 1) for r in (False, True)]) for s in shapes]
    assert any("stream" in f for f in fresh) and any("long" in f for f in fresh)

    def after(reverse):
        for s in fill:
            for d in (0, 1):
                for r in (False, True):
                    ops.launched_kernel(s, d, r)
        order = list(reversed(shapes)) if reverse else shapes
        got = [[asked(s, d, r, []) for d in (0, 1) for r in (False, True)] for s in order]
        return got[::-1] if reverse else got
    assert in_a_fresh_thread(lambda: after(False)) == fresh
    assert in_a_fresh_thread(lambda: after(True)) == fresh


@pytest.mark.parametrize("shape,named,launched", [((4096, 23, 7, 7), "plain", "stream"), ((64, 8, 56, 56), "tiled", "long"), ((2, 512, 7, 7), "register", "register"),
                                                  ((1024, 2048, 7, 7), "stream", "band"), ((64, 512, 7, 7), "register", "register")])
def test_the_queries_by_shape(shape, named, launched):
    assert ops.serving_kernel(shape, 0) == named and ops.launched_kernel(shape, 0) == launched
    assert ops.launched_kernel(shape, 0, aligned=False) == ops.serving_kernel(shape, 0, aligned=False)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,direction,residual,before", CALLS[:3])
def test_launches_it_with_the_same_bits(shape, direction, residual, before):
    d = make_inputs(shape, seed=4, loc=1.0, scale=2.0)

    def call(first):
        for b in first:
            for r in (False, True):
                ops.launched_kernel(b, 1, r)
        got, _ = run_fused(ops, d)
        return ops.last_kernel(), got
    (k0, a), (k1, b) = in_a_fresh_thread(lambda: call([])), in_a_fresh_thread(lambda: call(before))
    assert k0 == k1 == ops.launched_kernel(shape, 1)
    for k in a:
        assert (a[k] is None and b[k] is None) or np.array_equal(a[k], b[k]), k
    check_layer_own_mask(d, a, "%r " % (shape,))
