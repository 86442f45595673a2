"""Rows up to the longest that a call may have, 2^32 - 1 floats: the geometries of the masked form and of the kernel for long rows are
asked for without an overflow (the vectors of such a row, from the boundary below its start to the one above its end, hold more floats
than 32 bits count), and answer that they do not serve them."""
import ctypes
import subprocess
import sys

import pytest

QUERIES = """
import ctypes, sys
from anode_b200 import _lib
L, out, row = _lib.load(), (ctypes.c_uint32 * 7)(), int(sys.argv[1])
for d in (0, 1):
    for r in (0, 1):
        for query, most in ((L.anode_gpu_batch_norm_stream_masked_geometry, 0), (L.anode_gpu_batch_norm_long_geometry, 4 * 0x3fffffff)):
            vectors = row // 4 if row % 4 == 0 else (row + 6) // 4
            assert query(row, 1, 1, d, r, out) == 0 and out[0] == (vectors * 4 <= most), (query.__name__, d, r, list(out))
            assert not out[0] or out[3] == vectors
"""


@pytest.mark.parametrize("row", [2 ** 32 - n for n in range(1, 10)])
def test_geometries_of_the_longest_rows(row):
    # (in a process of its own: a division by zero ends one)
    p = subprocess.run([sys.executable, "-c", QUERIES, str(row)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, timeout=300)
    assert p.returncode == 0, p.stdout.decode()[-2000:]


@pytest.mark.parametrize("row", [1017, 1018, 1019, 1021, 1022, 1023, 1025])
def test_the_longest_rows_of_the_masked_form(row):
    # a block has a thread for each of up to 256 vectors
    from anode_b200 import _lib
    out = (ctypes.c_uint32 * 7)()
    assert _lib.load().anode_gpu_batch_norm_stream_masked_geometry(row, 1, 1, 0, 0, out) == 0
    assert out[0] == ((row + 6) // 4 <= 256)
