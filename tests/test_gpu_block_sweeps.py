"""SSOR sweeps by phases and blocks (sell.cu) against the oracle's V-cycle, where
the blocks' shapes can go wrong: ragged planes, one and three smoothing steps,
omega != 1 (no pass left out at a turn), 32-warp blocks (planes of more than
2,048 rows), blocks whose two passes do not fit shared memory together (FP64,
129^2 planes: one launch per pass), a colouring without blocks, and a pattern
that is not split (two coupled rows of one colour, possible when the pattern is
not symmetric).

Bars: FP64 within 1e-10 relative (max norm): the sums of a row are the same ones
in another order; FP32 within 1e-4 (FP32 values and iterates)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def vcycle_error(pmg, oracle, levels, colors, form=2, steps=2, omega=1.0, prec=0, matrices=None):
    import torch
    nl = len(levels)
    h = pmg.Handle(nl, pmg.default_params(precision=prec, pre_smooth=steps, post_smooth=steps, smooth_omega=omega))
    h.set_coefficients(pmg.coeff(kind=pmg.COEF_CONST, eps=1e-2, b=(1, .5, .25), f=1.0))
    pmg.load_hierarchy(h, levels, lattice_colors=colors)
    h.assemble(-1, form, copy_out=False)
    olev = []
    for l, L in enumerate(levels):
        if matrices and matrices[l] is not None:
            h.set_matrix(l, matrices[l])
        d = dict(N=L["N"], Na=L["active_bound"], rp=L["rowptr"], kc=L["kcol"], a=h.get_matrix(l))
        if colors:
            d.update(colors=L["colors"], n_colors=L["n_colors"])
        else:
            c, n = greedy(L)
            d.update(colors=c, n_colors=n)
        if l > 0:
            d["P"] = L["P"]
        olev.append(d)
    v = np.random.default_rng(5).standard_normal(levels[-1]["N"])
    vd = torch.tensor(v, dtype=torch.float64, device="cuda")
    zd = torch.empty_like(vd)
    h.vcycle(vd.data_ptr(), zd.data_ptr())
    torch.cuda.synchronize()
    zo = oracle.mg_apply(olev, v, pre=steps, post=steps, omega=omega, coarse_direct=True)
    h.close()
    return float(np.max(np.abs(zd.cpu().numpy() - zo)) / np.max(np.abs(zo)))


def greedy(L):
    """The library's greedy colouring of the active rows (in row order)."""
    rp, kc, na = L["rowptr"], L["kcol"], L["active_bound"]
    color = np.full(L["N"], -1, dtype=np.int32)
    for r in range(na):
        used = set(color[kc[rp[r]:rp[r + 1]]])
        c = 0
        while c in used:
            c += 1
        color[r] = c
    n = int(color.max()) + 1
    color[na:] = 0
    return color, n


@pytest.mark.parametrize("elem,n,nl,steps,omega,prec", [
    (1, 18, 2, 1, 1.0, 0),   # Q1: 2 phases of 4 colours, ragged planes of 19^2 nodes
    (1, 18, 2, 3, 0.9, 0),
    (2, 10, 2, 1, 0.8, 0),   # Q2: 3 phases of 9 colours, planes of 21^2 nodes
    (2, 10, 2, 3, 1.0, 1),
    (12, 14, 3, 2, 1.0, 0),  # P2 tetrahedra
    (1, 64, 4, 2, 1.0, 1),   # 4 colours of 32 slices per plane: 32-warp blocks
    (1, 64, 4, 1, 0.9, 0),
])
def test_block_sweeps_match_oracle(pmg, oracle, elem, n, nl, steps, omega, prec):
    levels = pmg.struct_hierarchy(elem, n, nl)
    err = vcycle_error(pmg, oracle, levels, True, form=1 if elem == 12 else 2, steps=steps, omega=omega, prec=prec)
    assert err < (1e-4 if prec else 1e-10), err


def test_blocks_too_large_for_two_passes(pmg, oracle):
    """129^2-node planes in FP64: iterate and second-pass start exceed shared memory together."""
    assert vcycle_error(pmg, oracle, pmg.struct_hierarchy(1, 128, 5), True) < 1e-10


@pytest.mark.parametrize("elem,n", [(1, 16), (2, 8)])
def test_greedy_colouring_matches_oracle(pmg, oracle, elem, n):
    """The library's own colouring of the same patterns, whatever blocks it has."""
    assert vcycle_error(pmg, oracle, pmg.struct_hierarchy(elem, n, 2), False) < 1e-10


def test_unsplit_pattern(pmg, oracle):
    """An entry (r, c) whose partner (c, r) is missing: the greedy colouring, which looks at row r when c is
    still uncoloured, gives both rows one colour, and the level's sweeps read whole rows.  The entry's value is
    0, so the order inside the colour does not matter."""
    levels = pmg.struct_hierarchy(1, 16, 2)
    F = levels[-1]
    rp, kc, na = F["rowptr"], F["kcol"], F["active_bound"]
    color, _ = greedy(F)
    r = 0
    c = next(j for j in range(1, na) if color[j] == color[r] and j not in set(kc[rp[r]:rp[r + 1]]))
    at = rp[r] + int(np.searchsorted(kc[rp[r]:rp[r + 1]], c))
    F["kcol"] = np.insert(kc, at, c).astype(np.int32)
    F["rowptr"] = (rp + (np.arange(rp.size) > r)).astype(np.int32)
    color2, _ = greedy(F)
    assert color2[r] == color2[c]
    assert vcycle_error(pmg, oracle, levels, False) < 1e-10
