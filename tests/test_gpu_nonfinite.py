"""A channel that holds a NaN or an infinity: its variance and its running variance become NaN, its output too, whichever
kernel serves the layer, and its neighbours are bit for bit what they are without it."""
import numpy as np
import pytest

from tests.test_gpu_fused import run_fused
from tests.util import make_inputs

pytestmark = pytest.mark.gpu

# register-resident kernel: teams of one warp, one block and several, 4-byte and 16-byte loads; streaming kernel; the rest forced
CASES = [("auto", (2, 512, 7, 7)), ("auto", (1, 53, 39, 25)), ("auto", (32, 64, 28, 28)), ("auto", (4, 16, 112, 112)),
         ("auto", (1411, 128, 7, 7)), ("auto", (2000, 20, 11, 11)), ("cluster", (64, 96, 7, 7)), ("cluster", (4, 4, 7, 7)),
         ("tiled", (16, 8, 56, 56)), ("tiled", (9, 5, 55, 55)), ("plain", (5, 3, 7, 7)), ("plain", (64, 96, 7, 7)),
         ("plain", (16, 8, 56, 56)), ("resident", (16, 8, 56, 56))]


@pytest.mark.parametrize("kernel,shape", CASES)
def test_a_poisoned_channel_has_no_variance(kernel, shape):
    from anode_b200 import ops
    ops.set_kernel(kernel)
    try:
        d = make_inputs(shape, seed=sum(shape), loc=0.5, scale=2.0)
        clean, _ = run_fused(ops, d)
        rng = np.random.default_rng(7)
        for place in ("first", "anywhere"):
            x = d["x"].copy()
            for c, v in ((0, np.nan), (2, np.inf)):
                row = x[:, c].reshape(-1).copy()
                row[0 if place == "first" else int(rng.integers(1, row.size))] = v
                x[:, c] = row.reshape(x[:, c].shape)
            got, ws = run_fused(ops, dict(d, x=x))
            for c in (0, 2):
                assert np.isnan(got["var"][c]) and np.isnan(got["run_var"][c]), (kernel, shape, place, c)
                assert not np.isfinite(got["mean"][c]) and not np.isfinite(got["run_mean"][c])
                assert np.isnan(got["y"][:, c]).all()
            rest = [c for c in range(shape[1]) if c not in (0, 2)]
            for k in ("mean", "var", "run_mean", "run_var", "dgamma", "dbeta"):
                assert np.array_equal(got[k][rest], clean[k][rest]), (kernel, shape, place, k)
            for k in ("y", "dx"):
                assert np.array_equal(got[k][:, rest], clean[k][:, rest]), (kernel, shape, place, k)
    finally:
        ops.set_kernel("auto")
