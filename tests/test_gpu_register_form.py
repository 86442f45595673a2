"""The register-resident kernel's form of fewer registers is launched where it makes one wave of blocks of what would be two, and only
there: by the blocks that the device holds of either form, not by a register count that a form does not have."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FWD, BWD, FWD_RES, BWD_RES = (0, 0), (1, 0), (0, 1), (1, 1)
KEYS = ["applies", "floats", "cluster", "blocks", "threads", "ordinary", "few", "dense"]


def form(shape, call):
    from anode_b200 import _lib
    out = (ctypes.c_uint32 * 8)()
    assert _lib.load().anode_gpu_batch_norm_register_form(int(np.prod(shape[2:])), shape[1], shape[0], call[0], call[1], out) == 0
    return dict(zip(KEYS, list(out)))


@pytest.mark.parametrize("shape,call,dense", [
    ((22, 328, 8, 8), BWD, 0), ((10, 912, 8, 8), BWD, 0), ((125, 1206, 2, 2), BWD, 0),
    ((16, 899, 6, 6), BWD, 0), ((225, 56, 8, 10), FWD, 1), ((3, 239, 1, 1451), FWD, 1), ((6, 278, 1, 354), FWD, 1), ((19, 1970, 1, 65), BWD_RES, 0), ((2, 512, 7, 7), BWD, 0)])
def test_form(shape, call, dense):
    assert form(shape, call)["dense"] == dense


def test_one_wave_in_the_place_of_two():
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(1)
    seen = set()
    for _ in range(3000):
        n, c, row = int(rng.integers(1, 300)), int(rng.integers(32, 2048)), int(rng.integers(2, 300))
        for call in (FWD, BWD, FWD_RES, BWD_RES):
            f = form((n, c, row), call)
            if not f["applies"] or f["floats"] > 8:
                assert not f["dense"]
                continue
            assert 1 <= f["ordinary"] <= f["few"] <= 2048 // f["threads"]
            num, den = {8: (9, 10), 4: (15, 16)}.get(f["cluster"], (1, 1))
            if call == BWD_RES:                        # (gains by it in one wave, too: as if the ordinary form had 64 registers)
                f["ordinary"] = min(f["ordinary"], 1024 // f["threads"])
            ordinary, few = (f[k] * sms * num // den for k in ("ordinary", "few"))
            assert f["dense"] == (f["blocks"] >= 128 and ordinary < f["blocks"] <= few * 21 // 20), (n, c, row, call, f)
            seen.add((call, f["dense"], f["floats"]))
    assert len(seen) == 16
