"""A pattern that couples two rows of one colour (possible for an unsymmetric one:
the greedy colouring looks at row r while its column c is still uncoloured): an
update of that colour directly after another one changes x, so no update may be
left out where the sweeps turn.  Row r = 0 takes x_c of a row c > r in its own colour.

Every colour has at most 32 rows, hence one slice, whose rows are all formed from
the values before the update: the same as the oracle's order by rows inside a
colour, because c > r.  The coupled colour is the first one (row 0's), updated twice
where a second step follows a backward sweep.  Bar: 1e-10 relative (max norm, FP64)."""
import numpy as np
import pytest

from test_gpu_dirichlet_rows import greedy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("elem,n,steps,omega", [(1, 4, 2, 1.0), (1, 4, 3, 1.0), (1, 4, 2, 0.9)])
def test_repeated_colour_is_not_left_out(pmg, oracle, elem, n, steps, omega):
    import torch
    levels = pmg.struct_hierarchy(elem, n, 2)
    F = levels[1]
    rp, kc, na = F["rowptr"], F["kcol"], F["active_bound"]
    color, _ = greedy(F)
    r = 0
    c = next(j for j in range(1, na) if color[j] == color[r] and j not in set(kc[rp[r]:rp[r + 1]]))
    at = rp[r] + int(np.searchsorted(kc[rp[r]:rp[r + 1]], c))
    F["kcol"] = np.insert(kc, at, c).astype(np.int32)
    F["rowptr"] = (rp + (np.arange(rp.size) > r)).astype(np.int32)
    color, _ = greedy(F)
    assert color[r] == color[c] and np.bincount(color[:na]).max() <= 32
    h = pmg.Handle(2, pmg.default_params(precision=pmg.PREC_FP64, pre_smooth=steps, post_smooth=steps,
                                         smooth_omega=omega))
    h.set_coefficients(pmg.coeff(kind=pmg.COEF_CONST, eps=1e-2, b=(1, .5, .25), f=1.0))
    pmg.load_hierarchy(h, levels, lattice_colors=False)
    h.assemble(-1, pmg.FORM_SUPG, copy_out=False)
    a = h.get_matrix(1)
    a[at] = 0.5 * np.max(np.abs(a[F["rowptr"][r]:F["rowptr"][r + 1]]))
    h.set_matrix(1, a)
    olev = []
    for l, L in enumerate(levels):
        colors, nc = greedy(L)
        olev.append(dict(N=L["N"], Na=L["active_bound"], rp=L["rowptr"], kc=L["kcol"], a=h.get_matrix(l),
                         colors=colors, n_colors=nc))
    olev[1]["P"] = F["P"]
    v = np.random.default_rng(n).standard_normal(F["N"])
    vd = torch.tensor(v, dtype=torch.float64, device="cuda")
    zd = torch.empty_like(vd)
    h.vcycle(vd.data_ptr(), zd.data_ptr())
    torch.cuda.synchronize()
    h.close()
    zo = oracle.mg_apply(olev, v, pre=steps, post=steps, omega=omega, coarse_direct=True)
    err = np.max(np.abs(zd.cpu().numpy() - zo)) / np.max(np.abs(zo))
    assert err < 1e-10, err
