"""Device memory of the solve copies: what only the sweeps read (kept sums, base
vector, the blocks' copy of the entries inside them) is there only in the precision
and for the smoother that sweeps.  Q2 32^3, finest level 275 k rows: the entries
inside the blocks are those between active rows of one phase (nine colours)."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def inside_entries(L):
    na, phase = L["active_bound"], np.asarray(L["colors"]) // 9
    rows = np.repeat(np.arange(L["N"]), np.diff(L["rowptr"]))
    act = (rows < na) & (L["kcol"] < na)
    r, c = rows[act], L["kcol"][act]
    return int(np.count_nonzero((phase[r] == phase[c]) & (r != c)))


CHILD = r"""
import ctypes, json, sys
sys.path.insert(0, {root!r})
import torch
import parmoon_b200 as P


def used():
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


levels = P.struct_hierarchy(2, 32, 4)
h = P.Handle(4, P.default_params(precision=P.PREC_FP32, smoother={smoother}, smooth_omega=0.5, lin_maxit=2))
h.set_coefficients(P.coeff(kind=P.COEF_CONST, eps=1.0, b=(1, .5, .25), f=1.0))
P.load_hierarchy(h, levels)
h.assemble(-1, P.FORM_GALERKIN, copy_out=False)
u = [used()]
assert h.solve(raise_on_error=False)[2] in (0, -4)
u.append(used())
sec = ctypes.c_double()
assert P.lib().pmg_time_kernel(h.h, 2, 3, 0, 1, ctypes.byref(sec), None, None) == 0  # FP64 SSOR steps
u.append(used())
h.assemble(-1, P.FORM_GALERKIN, copy_out=False)
assert h.solve(raise_on_error=False)[2] in (0, -4)
u.append(used())
print(json.dumps([b - a for a, b in zip(u, u[1:])]))
"""


def growth(smoother):
    """Bytes taken by a solve, by FP64 sweeps after it, by a second solve; in a process of its own
    (what a handle gives back need not show while its process lives)."""
    p = subprocess.run([sys.executable, "-c", CHILD.format(root=ROOT, smoother=smoother)], capture_output=True, text=True,
                       timeout=300)
    assert p.returncode == 0, p.stderr[-3000:]
    return json.loads(p.stdout.strip().splitlines()[-1])


def test_only_what_sweeps_is_held(pmg):
    inside = inside_entries(pmg.struct_hierarchy(2, 32, 4)[-1])
    assert 4 * inside > 12 << 20  # well above the granularity of device allocations
    jacobi, ssor = growth(pmg.SMOOTHER_JACOBI), growth(pmg.SMOOTHER_SSOR)
    # a Jacobi smoother holds no blocks
    assert jacobi[0] <= ssor[0] - 3.5 * inside, (jacobi, ssor, inside)
    # an FP32 V-cycle none in FP64: they come when FP64 sweeps are asked for
    assert ssor[1] >= 7 * inside, (ssor, inside)
    # and a second solve takes nothing more
    assert ssor[2] <= 4 << 20, ssor
