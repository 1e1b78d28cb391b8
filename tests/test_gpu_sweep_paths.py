"""Which way an SSOR step takes, seen from the number of its kernel launches: by
phases and blocks (a product and a sweep per phase), or one launch per colour
(2 n - 1 of them for n colours: the turn is done once), and that a level is not
swept by blocks where the largest block, one CTA's work, takes longer than the
colours.  Then the sweeps whose two passes at a turn do not fit shared memory
together (a launch each), against the oracle's V-cycle: a 64-colour lattice with
planes of 160^2 nodes in FP32 and of 116^2 in FP64.  Bars as test_gpu_block_sweeps.py:
1e-10 (FP64), 1e-4 (FP32)."""
import ctypes

import numpy as np
import pytest

from test_gpu_dirichlet_rows import greedy

pytestmark = pytest.mark.gpu


def step_launches(pmg, h, level, prec):
    """Kernel launches of one SSOR step on an arbitrary x."""
    def total(reps):
        n0, n1, sec = ctypes.c_ulonglong(), ctypes.c_ulonglong(), ctypes.c_double()
        pmg.lib().pmg_launch_count(ctypes.byref(n0))
        assert pmg.lib().pmg_time_kernel(h.h, 3 if prec else 2, level, 0, reps, ctypes.byref(sec), None, None) == 0
        pmg.lib().pmg_launch_count(ctypes.byref(n1))
        return n1.value - n0.value
    total(1)  # (the solve copy is built)
    return total(2) - total(1)


def lattice(nx, ny, nz, offsets, mod):
    """Pattern of the offsets on an nx x ny x nz lattice, all rows active, colours by the residues modulo mod."""
    n = nx * ny * nz
    idx = np.arange(n)
    i, j, k = idx % nx, idx // nx % ny, idx // (nx * ny)
    keys = []
    for di, dj, dk in offsets:
        ok = (i + di >= 0) & (i + di < nx) & (j + dj >= 0) & (j + dj < ny) & (k + dk >= 0) & (k + dk < nz)
        keys.append(idx[ok] * n + (idx + di + nx * (dj + ny * dk))[ok])
    key = np.sort(np.concatenate(keys))
    rp = np.concatenate([[0], np.cumsum(np.bincount(key // n, minlength=n))]).astype(np.int32)
    return rp, (key % n).astype(np.int32), ((i % mod) + mod * ((j % mod) + mod * (k % mod))).astype(np.int32)


BOX = [(a, b, c) for c in (-1, 0, 1) for b in (-1, 0, 1) for a in (-1, 0, 1)]
STAR = [(0, 0, 0)] + [tuple(s * (d == k) for k in range(3)) for d in range(3) for s in (-1, 1)]


def one_level(pmg, rp, kc, colors, n_colors):
    h = pmg.Handle(1, pmg.default_params())
    n = rp.size - 1
    h.set_level_csr(0, rp, kc, n)
    h.set_row_colors(0, colors, n_colors)
    h.set_matrix(0, np.where(np.repeat(np.arange(n), np.diff(rp)) == kc, 2.0 * np.diff(rp).max(), -1.0))
    return h


@pytest.mark.parametrize("elem,n,expect", [(1, 32, 6), (2, 16, 10), (12, 16, 10), (1, 64, 6)])
@pytest.mark.parametrize("prec", [0, 1])
def test_lattice_colours_have_blocks(pmg, elem, n, expect, prec):
    """2 phases of 4 colours: 3 products and 3 sweeps; 3 phases of 9: 5 and 5."""
    L = pmg.struct_hierarchy(elem, n, 1)[0]
    h = pmg.Handle(1, pmg.default_params())
    h.set_level_csr(0, L["rowptr"], L["kcol"], L["active_bound"])
    h.set_row_colors(0, L["colors"], L["n_colors"])
    rows = np.repeat(np.arange(L["N"]), np.diff(L["rowptr"]))
    h.set_matrix(0, np.where(rows == L["kcol"], 200.0, -1.0))
    assert step_launches(pmg, h, 0, prec) == expect
    h.close()


@pytest.mark.parametrize("prec", [0, 1])
def test_greedy_colours_of_q2_have_none(pmg, prec):
    L = pmg.struct_hierarchy(2, 8, 1)[0]
    _, n = greedy(L)
    h = pmg.Handle(1, pmg.default_params())
    h.set_level_csr(0, L["rowptr"], L["kcol"], L["active_bound"])
    rows = np.repeat(np.arange(L["N"]), np.diff(L["rowptr"]))
    h.set_matrix(0, np.where(rows == L["kcol"], 200.0, -1.0))
    assert step_launches(pmg, h, 0, prec) == 2 * n - 1
    h.close()


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("nx,ny,nz", [(129, 129, 9), (201, 201, 9)])
def test_thin_domains_go_by_colours(pmg, nx, ny, nz, prec):
    h = one_level(pmg, *lattice(nx, ny, nz, BOX, 2), 8)
    assert step_launches(pmg, h, 0, prec) == 15
    h.close()


@pytest.mark.parametrize("prec", [0, 1])
def test_unbalanced_blocks_go_by_colours(pmg, prec):
    """One large component and three small ones in each phase."""
    parts = [lattice(151, 151, 2, BOX, 2)] + [lattice(5, 5, 2, BOX, 2)] * 3
    rp, kc, colors, n, nnz = [np.zeros(1, np.int32)], [], [], 0, 0
    for r, k, c in parts:
        rp.append((r[1:] + nnz).astype(np.int32))
        kc.append((k + n).astype(np.int32))
        colors.append(c)
        n, nnz = n + c.size, nnz + k.size
    h = one_level(pmg, np.concatenate(rp), np.concatenate(kc), np.concatenate(colors), 8)
    assert step_launches(pmg, h, 0, prec) == 15
    h.close()


def test_coupled_colour_goes_by_colours_twice_at_the_turn(pmg):
    rp, kc, colors = lattice(20, 20, 20, BOX, 2)
    kc = np.insert(kc, rp[1], 2 + 20 * (10 + 20 * 10)).astype(np.int32)  # row 0 with a row of its own colour
    rp = (rp + (np.arange(rp.size) > 0)).astype(np.int32)
    row = kc[rp[0]:rp[1]]
    assert np.all(np.diff(row) > 0) and colors[row[-1]] == colors[0]
    h = pmg.Handle(1, pmg.default_params())
    h.set_level_csr(0, rp, kc, rp.size - 1)
    n = len(set(colors_of(rp, kc)))
    rows = np.repeat(np.arange(rp.size - 1), np.diff(rp))
    h.set_matrix(0, np.where(rows == kc, 60.0, -1.0))
    assert step_launches(pmg, h, 0, 0) == 2 * n
    h.close()


def colors_of(rp, kc):
    c, _ = greedy(dict(rowptr=rp, kcol=kc, active_bound=rp.size - 1, N=rp.size - 1))
    return c


@pytest.mark.parametrize("side,prec", [(160, 1), (116, 0)])
def test_turn_in_two_launches(pmg, oracle, side, prec):
    """4 phases of 16 colours; 7 products, 7 sweeps and one more at the turn."""
    import torch
    rp, kc, colors = lattice(side, side, 16, STAR, 4)
    n, nc = rp.size - 1, 512
    rng = np.random.default_rng(side)
    rows = np.repeat(np.arange(n), np.diff(rp))
    a = np.where(rows == kc, 7.0, rng.uniform(-1, 0, kc.size))
    # a small coarse level of its own: tridiagonal, every fine row from one coarse row
    crp = np.concatenate([[0], np.cumsum([2] + [3] * (nc - 2) + [2])]).astype(np.int32)
    ckc = np.concatenate([[c + d for d in (-1, 0, 1) if 0 <= c + d < nc] for c in range(nc)]).astype(np.int32)
    ca = np.where(np.repeat(np.arange(nc), np.diff(crp)) == ckc, 800.0, -300.0)
    P = (np.arange(n + 1, dtype=np.int32), (np.arange(n) * nc // n).astype(np.int32), rng.uniform(0.5, 1, n))
    h = pmg.Handle(2, pmg.default_params(precision=prec))
    h.set_level_csr(0, crp, ckc, nc)
    h.set_level_csr(1, rp, kc, n)
    h.set_row_colors(1, colors, 64)
    h.set_transfer(1, *P, nc)
    h.set_matrix(0, ca)
    h.set_matrix(1, a)
    assert step_launches(pmg, h, 1, prec) == 15
    v = rng.standard_normal(n)
    vd = torch.tensor(v, dtype=torch.float64, device="cuda")
    zd = torch.empty_like(vd)
    torch.cuda.synchronize()
    h.vcycle(vd.data_ptr(), zd.data_ptr())
    torch.cuda.synchronize()
    h.close()
    cc = (np.arange(nc) % 2).astype(np.int32)
    zo = oracle.mg_apply([dict(N=nc, Na=nc, rp=crp, kc=ckc, a=ca, colors=cc, n_colors=2),
                          dict(N=n, Na=n, rp=rp, kc=kc, a=a, colors=colors, n_colors=64, P=P)], v, coarse_direct=True)
    err = np.max(np.abs(zd.cpu().numpy() - zo)) / np.max(np.abs(zo))
    assert err < (1e-4 if prec else 1e-10), err


@pytest.mark.parametrize("first", [0, 1])
def test_layout_follows_the_precision_in_use(pmg, first):
    """65 x 65 x 13 nodes, 8 colours: blocks are the faster way in FP32 only.  A level first used in
    FP64 is not laid out by blocks at all, one first used in FP32 is, and FP64 sweeps go by colours in both."""
    rp, kc, colors = lattice(65, 65, 13, BOX, 2)
    n = rp.size - 1
    h = pmg.Handle(1, pmg.default_params(precision=first))
    h.set_level_csr(0, rp, kc, n)
    h.set_row_colors(0, colors, 8)
    h.set_matrix(0, np.where(np.repeat(np.arange(n), np.diff(rp)) == kc, 60.0, -1.0))
    assert step_launches(pmg, h, 0, first) == (6 if first else 15)
    assert step_launches(pmg, h, 0, 1 - first) == 15
    h.close()
