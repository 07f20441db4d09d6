"""A table that the bin tiles refuse is an error of the call, also where a worker
thread finds it (in a process of its own: an exception that leaves a thread ends
the process)."""
import os
import subprocess
import sys

import pytest

SCRIPT = """
import numpy as np
from dioptrin_b200 import _native as N
rows = {rows}
rp = np.arange(rows + 1, dtype=np.int64)
rp[rows // 2 + 1:] += 1 << 27  # one bin of more than 2^27 entries
col = np.zeros(int(rp[-1]), np.int32)  # never read for that bin
counts = np.zeros(5, np.int64)
st = N.lib().dg_test_bin_items(8, rows, rp.ctypes.data, col.ctypes.data, counts.ctypes.data,
                               *[None] * 5)
assert st == N.DG_UNSUPPORTED and "too large" in N.last_error(), (st, N.last_error())
print("refused")
"""


@pytest.mark.parametrize("rows", [1, 400])  # one tile, and more tiles than threads
def test_a_bin_too_large_is_refused(rows):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(rows=rows)], capture_output=True,
                       text=True, timeout=120, cwd=root)
    assert r.returncode == 0 and "refused" in r.stdout, (r.returncode, r.stderr[-500:])
