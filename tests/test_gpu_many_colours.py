"""A level whose every row has a colour of its own (a lexicographic sweep): building
its solve copy takes host memory in proportion to the rows.  200,000 rows, diagonal
only; the tables are about 60 integers per row with a slice of 32 lanes for each,
200,000 x 60 x 4 bytes = 48 MB; bar 600 MB (a number per pair of a phase's blocks
and colours would be 2.8 GB)."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, json, resource, sys
sys.path.insert(0, {root!r})
import numpy as np
import parmoon_b200 as P
N = 200000
h = P.Handle(1, P.default_params())
h.set_level_csr(0, np.arange(N + 1), np.arange(N), N)
h.set_row_colors(0, np.arange(N), N)
h.set_matrix(0, np.full(N, 2.0))
before = resource.getrusage(resource.RUSAGE_SELF).ru_maxrss
sec = ctypes.c_double()
rc = P.lib().pmg_time_kernel(h.h, 1, 0, 0, 1, ctypes.byref(sec), None, None)
print(json.dumps(dict(rc=rc, mb=(resource.getrusage(resource.RUSAGE_SELF).ru_maxrss - before) / 1024)))
"""


def test_host_memory_in_proportion_to_the_rows():
    p = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-3000:]
    r = json.loads(p.stdout.strip().splitlines()[-1])
    assert r["rc"] == 0 and r["mb"] < 600, r
