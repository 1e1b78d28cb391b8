"""The coarsest level's inverse is no further from the exact one than LU with
partial pivoting and substitution is.  One FP64 cycle of a one-level handle on
the unit vector e_j returns column j of the inverse as it is (all other terms of
the product are 0).  The exact inverse: Newton steps in 64-bit-mantissa arithmetic
(numpy longdouble) from LAPACK's, until the correction is below 1e-18.  Active
rows 27 to 729 (tiles of 64 and a remainder, panels of 24 and a remainder).

Bar: |X - A^-1|_F <= |X_lu - A^-1|_F with LAPACK's LU and substitution.  Expected:
a Newton step leaves the rounding of X's entries, about 2^-54 each on average, LU a
few times 2^-53; exchange steps alone are above LU."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("elem,n,eps", [(1, 4, 1e-3), (1, 7, 1e-2), (1, 9, 1.0), (2, 4, 1e-3), (2, 5, 1e-3)])
def test_no_further_off_than_lu(pmg, elem, n, eps):
    import scipy.linalg
    import torch
    L = pmg.struct_hierarchy(elem, n, 1)[0]
    h = pmg.Handle(1, pmg.default_params(precision=pmg.PREC_FP64))
    h.set_coefficients(pmg.coeff(kind=pmg.COEF_CONST, eps=eps, b=(1, .5, .25), f=1.0))
    pmg.load_hierarchy(h, [L])
    h.assemble(0, pmg.FORM_SUPG, copy_out=False)
    na = L["active_bound"]
    D = np.zeros((L["N"], L["N"]))
    D[np.repeat(np.arange(L["N"]), np.diff(L["rowptr"])), L["kcol"]] = h.get_matrix(0)
    A = D[:na, :na]
    X = np.empty((na, na))
    vd = torch.zeros(L["N"], dtype=torch.float64, device="cuda")
    zd = torch.empty_like(vd)
    for j in range(na):
        vd[j] = 1.0
        torch.cuda.synchronize()  # (the handle's stream does not wait for torch's)
        h.vcycle(vd.data_ptr(), zd.data_ptr())
        X[:, j] = zd[:na].cpu().numpy()
        vd[j] = 0.0
    h.close()
    lu = scipy.linalg.lu_solve(scipy.linalg.lu_factor(A), np.eye(na))
    Al, ref = A.astype(np.longdouble), np.linalg.inv(A).astype(np.longdouble)
    for _ in range(4):
        step = ref @ (np.eye(na, dtype=np.longdouble) - Al @ ref)
        ref = ref + step
        if np.max(np.abs(step)) < 1e-18 * np.max(np.abs(ref)):
            break
    err = float(np.linalg.norm((X - ref).astype(np.float64)))
    err_lu = float(np.linalg.norm((lu - ref).astype(np.float64)))
    assert err <= err_lu, (err / err_lu, err_lu)
