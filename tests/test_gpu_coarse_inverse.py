"""The coarsest level's inverse (blocked Gauss-Jordan with partial pivoting): one
FGMRES iteration of a one-level handle is then a direct solve.  Active rows 1,
8 (one short panel), 27 (a panel of 24 and one of 3), 343, 729; and a matrix
whose diagonal is tiny, so that every pivot comes from another row.

Bars: |x - x_ref| <= 1e-12 |x_ref| (condition numbers below 1e3 and 1e4:
n eps cond = 729 * 2.2e-16 * 1e3 = 1.6e-10 bounds the error, the usual growth is
far smaller); a zero row is PMG_ERR_SINGULAR."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def level(pmg, n, elem=1):
    L = pmg.struct_hierarchy(elem, n, 1)[0]
    h = pmg.Handle(1, pmg.default_params(lin_maxit=1, restart=2, lin_red=1e-30))
    h.set_coefficients(pmg.coeff(kind=pmg.COEF_CONST, eps=1e-3, b=(1, .5, .25), f=1.0))
    pmg.load_hierarchy(h, [L], dirichlet=lambda x, y, z: 1.0 + x)
    h.assemble(0, pmg.FORM_SUPG, copy_out=False)
    return h, L


def dense(L, a):
    D = np.zeros((L["N"], L["N"]))
    D[np.repeat(np.arange(L["N"]), np.diff(L["rowptr"])), L["kcol"]] = a
    return D


@pytest.mark.parametrize("elem,n", [(1, 2), (1, 3), (1, 4), (2, 4), (2, 5)])
@pytest.mark.parametrize("permuted", [False, True])
def test_one_cycle_is_a_direct_solve(pmg, elem, n, permuted):
    h, L = level(pmg, n, elem)
    a = h.get_matrix(0)
    na = L["active_bound"]
    if permuted:  # couplings of size 1, diagonal 1e-9: well conditioned only through pivoting
        rng = np.random.default_rng(n)
        rows = np.repeat(np.arange(L["N"]), np.diff(L["rowptr"]))
        act = rows < na
        a[act] = rng.uniform(-1, 1, act.sum())
        a[act & (L["kcol"] == rows)] = 1e-9
        h.set_matrix(0, a)
    D = dense(L, a)
    if permuted and (na == 1 or np.linalg.cond(D) > 1e4):
        pytest.skip("no well-conditioned matrix of this shape")
    b = np.random.default_rng(1).standard_normal(L["N"])
    x, _, _ = h.solve(sol=np.zeros(L["N"]), rhs=b, raise_on_error=False)
    ref = np.linalg.solve(D, b)
    assert np.linalg.norm(x - ref) <= 1e-12 * np.linalg.norm(ref)
    h.close()


def test_zero_row_is_singular(pmg):
    h, L = level(pmg, 4)
    a = h.get_matrix(0)
    a[L["rowptr"][5]:L["rowptr"][6]] = 0.0
    h.set_matrix(0, a)
    _, _, rc = h.solve(raise_on_error=False)
    assert rc == -8
    h.close()
