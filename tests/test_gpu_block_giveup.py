"""The bounded waits of the block sweeps: with every wait expecting one more slice
than there is (PMG_TEST_BLK_EXTRA), each of them runs out after about 0.2 s, the
launches end, and the call reports PMG_ERR_STATE; the flag is cleared, and the next
call on the same handle and context works.  Two levels, Q1 18^3 on the finer one
(phases and blocks), as child processes."""
import json
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SETUP = r"""
import ctypes, json, os, sys
os.environ["PMG_NO_GRAPH"] = "1"  # launch the V-cycle kernels directly, so the test switch is read per launch
sys.path.insert(0, {root!r})
import parmoon_b200 as P
levels = P.struct_hierarchy(1, 18, 2)
h = P.Handle(2, P.default_params(precision={prec}, lin_maxit=1, pre_smooth=1, post_smooth=1))
h.set_coefficients(P.coeff(kind=P.COEF_CONST, eps=1e-2, b=(1.0, 0.5, 0.25), f=1.0))
P.load_hierarchy(h, levels, dirichlet=lambda x, y, z: (abs(x) < 1e-12).astype(float))
h.assemble(-1, P.FORM_SUPG, copy_out=False)
os.environ["PMG_TEST_BLK_EXTRA"] = "1"
{fail}
del os.environ["PMG_TEST_BLK_EXTRA"]
h.set_params(P.default_params(precision={prec}))
_, st, rc_ok = h.solve(raise_on_error=False)
print(json.dumps(dict(rc_fail=rc_fail, rc_ok=rc_ok, rel=st.rel_res, its=st.iterations)))
"""

SOLVE = "_, st, rc_fail = h.solve(raise_on_error=False)"


def run(prec, fail):
    p = subprocess.run([sys.executable, "-c", SETUP.format(root=ROOT, prec=prec, fail=fail)], capture_output=True,
                       text=True, timeout=300)
    assert p.returncode == 0, p.stderr[-3000:]
    return json.loads(p.stdout.strip().splitlines()[-1])


@pytest.mark.parametrize("prec", [0, 1])
def test_solve_gives_up_and_recovers(prec):
    r = run(prec, SOLVE)
    assert r["rc_fail"] == -3, r
    assert r["rc_ok"] == 0 and r["rel"] <= 1e-10, r


TIMED = r"""
sec = ctypes.c_double()
rc_fail = P.lib().pmg_time_kernel(h.h, {kernel}, 1, P.FORM_SUPG, 1, ctypes.byref(sec), None, None)
"""


@pytest.mark.parametrize("prec,kernel", [(0, 2), (1, 3)])
def test_timed_sweep_reports_and_clears(prec, kernel):
    """pmg_time_kernel runs the same sweeps: it reports what gave up, and leaves no
    flag behind for the next solve."""
    r = run(prec, TIMED.format(kernel=kernel))
    assert r["rc_fail"] == -3, r
    assert r["rc_ok"] == 0 and r["rel"] <= 1e-10, r
