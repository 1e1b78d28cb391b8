"""A caller's pattern and matrix (pmg_set_matrix) whose Dirichlet rows hold more
than the diagonal (the reference's own hold the diagonal only): the V-cycle's defect on these rows is f_D - A_Da x_a - A_DD x_D, and a
transfer that couples Dirichlet dofs of the fine level to active dofs of the
coarse one (the cell averages of the non-conforming elements do; for the others the
test adds such weights) takes it into the coarse right-hand side.

Levels whose sweeps run by blocks, by colours and as whole rows, one and two
smoothing steps, against the oracle's V-cycle.  Bars: FP64 within 1e-10 relative
(max norm), FP32 within 1e-4 (FP32 values and iterates)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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


@pytest.mark.parametrize("elem,n,lattice,smoother,steps,prec", [
    (3, 12, False, 3, 2, 0),   # non-conforming, its own transfer
    (3, 12, False, 3, 1, 1),
    (1, 18, True, 3, 1, 0),    # Q1, phases and blocks
    (1, 18, False, 3, 2, 0),
    (2, 10, True, 3, 2, 1),    # Q2, phases and blocks
    (1, 18, True, 2, 2, 0),    # SOR: the defect over whole rows
])
def test_defect_of_full_dirichlet_rows(pmg, oracle, elem, n, lattice, smoother, steps, prec):
    import torch
    elem = pmg.NQ1_HEX if elem == 3 else elem
    levels = pmg.struct_hierarchy(elem, n, 2)
    F, C = levels[1], levels[0]
    na, nf = F["active_bound"], F["N"]
    rng = np.random.default_rng(n + elem)
    # Dirichlet rows coupled to the cells' other dofs
    rows, cols = [np.repeat(np.arange(nf), np.diff(F["rowptr"]))], [F["kcol"]]
    ed = F["elem_dof"].reshape(n ** 3, -1)
    for a in range(ed.shape[1]):
        on = ed[:, a] >= na
        rows.append(np.repeat(ed[on, a], ed.shape[1]))
        cols.append(ed[on].reshape(-1))
    key = np.unique(np.concatenate(rows).astype(np.int64) * nf + np.concatenate(cols))
    F["rowptr"] = np.concatenate([[0], np.cumsum(np.bincount(key // nf, minlength=nf))]).astype(np.int32)
    F["kcol"] = (key % nf).astype(np.int32)
    if elem != pmg.NQ1_HEX:
        # one more weight per Dirichlet row, on an active coarse dof
        rp, col, val = F["P"]
        rows = np.repeat(np.arange(nf), np.diff(rp))
        extra = rng.integers(0, C["active_bound"], nf - na)
        rows = np.concatenate([rows, np.arange(na, nf)])
        col, val = np.concatenate([col, extra]), np.concatenate([val, rng.uniform(0.1, 0.5, nf - na)])
        o = np.argsort(rows, kind="stable")
        F["P"] = (np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=nf))]).astype(np.int32),
                  col[o].astype(np.int32), val[o])
    h = pmg.Handle(2, pmg.default_params(precision=prec, smoother=smoother, pre_smooth=steps, post_smooth=steps))
    h.set_coefficients(pmg.coeff(kind=pmg.COEF_CONST, eps=1e-2, b=(1, .5, .25), f=1.0))
    pmg.load_hierarchy(h, levels, lattice_colors=lattice)
    h.assemble(-1, pmg.FORM_SUPG, copy_out=False)
    a = h.get_matrix(1)
    scale = np.max(np.abs(a[:F["rowptr"][na]]))
    a[F["rowptr"][na]:] = rng.uniform(-scale, scale, a.size - F["rowptr"][na])
    h.set_matrix(1, a)
    olev = []
    for l, L in enumerate(levels):
        colors, nc = (L["colors"], L["n_colors"]) if lattice else greedy(L)
        olev.append(dict(N=L["N"], Na=L["active_bound"], rp=L["rowptr"], kc=L["kcol"], a=h.get_matrix(l),
                         colors=colors, n_colors=nc))
    olev[1]["P"] = F["P"]
    v = rng.standard_normal(nf)
    v[na:] = 0.0
    vd = torch.tensor(v, dtype=torch.float64, device="cuda")
    zd = torch.empty_like(vd)
    h.vcycle(vd.data_ptr(), zd.data_ptr())
    torch.cuda.synchronize()
    h.close()
    zo = oracle.mg_apply(olev, v, pre=steps, post=steps, smoother=smoother, coarse_direct=True)
    err = np.max(np.abs(zd.cpu().numpy() - zo)) / np.max(np.abs(zo))
    assert err < (1e-4 if prec else 1e-10), err
