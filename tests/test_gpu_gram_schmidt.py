"""The Arnoldi columns of FGMRES(m): all inner products of a column are taken at
once and corrected to modified Gram-Schmidt by the products of the basis vectors.

Oracle: FGMRES(m) written out here in numpy with step-by-step modified
Gram-Schmidt, on the device's matrix and V-cycle (a weak one, so that the larger
restarts fill).  Both minimise the same residual; rounding moves it by about
m * eps * cond(H) * res0, far below the 1e-9 res0 allowed, while a wrong
coefficient in any column leaves a residual of another size.  Restarts below, at
and above one and two groups of eight vectors, and the largest one."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def fgmres_residual(A, M, b, x, m):
    r = b - A @ x
    beta = np.linalg.norm(r)
    V, Z, H = [r / beta], [], np.zeros((m + 1, m))
    for i in range(m):
        Z.append(M(V[i]))
        w = A @ Z[i]
        for k in range(i + 1):
            H[k, i] = w @ V[k]
            w = w - H[k, i] * V[k]
        H[i + 1, i] = np.linalg.norm(w)
        V.append(w / H[i + 1, i])
    y = np.linalg.lstsq(H, np.r_[beta, np.zeros(m)], rcond=None)[0]
    return beta, np.linalg.norm(b - A @ (x + np.array(Z).T @ y))


@pytest.mark.parametrize("n,levels,restart", [(4, 2, 1), (4, 2, 7), (4, 2, 8), (12, 3, 9), (16, 3, 17), (4, 2, 33), (8, 2, 60)])
def test_residual_of_a_full_restart(pmg, n, levels, restart):
    import torch
    prm = pmg.default_params(precision=pmg.PREC_FP64, restart=restart, lin_maxit=restart, lin_red=1e-30,
                             lin_res_min=1e-30, smoother=pmg.SMOOTHER_JACOBI, smooth_omega=0.05,
                             coarse_smoother=pmg.COARSE_JACOBI, coarse_maxit=1, pre_smooth=1, post_smooth=0)
    lv = pmg.struct_hierarchy(pmg.Q1_HEX, n, levels, jitter=0.0, seed=1)
    h = pmg.Handle(levels, prm)
    h.set_coefficients(pmg.coeff(kind=pmg.COEF_CONST, eps=0.05, b=(1.0, 0.5, 0.25), c=1.0, f=1.0))
    pmg.load_hierarchy(h, lv)
    h.assemble(-1, pmg.FORM_SUPG, copy_out=False)
    F = lv[-1]
    A = sp.csr_matrix((h.get_matrix(levels - 1), F["kcol"], F["rowptr"]))
    b = h.get_rhs(levels - 1)
    x0 = np.zeros_like(b)
    x0[F["active_bound"]:] = b[F["active_bound"]:]

    def M(v):
        vd, zd = torch.from_numpy(v.copy()).cuda(), torch.zeros(len(v), dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        h.vcycle(vd.data_ptr(), zd.data_ptr())
        torch.cuda.synchronize()
        return zd.cpu().numpy()

    runs = [h.solve(sol=np.zeros_like(b), rhs=b, raise_on_error=False) for _ in range(2)]
    assert np.array_equal(runs[0][0], runs[1][0])  # the sums are added in a fixed order
    st = runs[0][1]
    assert st.iterations == restart
    res0, ref = fgmres_residual(A, M, b, x0, restart)
    assert abs(st.res0 - res0) <= 1e-12 * res0
    assert ref < res0
    assert abs(st.res_final - ref) <= 1e-9 * res0
    h.close()
