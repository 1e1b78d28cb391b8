"""The coefficient table is checked and put into element order on the device: a
non-finite value anywhere is refused and leaves the level's table as it was."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("elem,n0,rule,other", [("Q1_HEX", 2, "GAUSS2", "GAUSS3"), ("P2_TET", 1, "KEAST11", "KEAST5"),
                                                ("Q2_HEX", 5, "GAUSS3", "GAUSS4")])
def test_nonfinite_table_is_refused_and_the_old_one_kept(pmg, elem, n0, rule, other):
    fm = pmg.FORM_GALERKIN
    levels = pmg.struct_hierarchy(getattr(pmg, elem), n0, 1, jitter=0.0, seed=1)
    prm = pmg.default_params(quad_rule=getattr(pmg, "QUAD_" + rule))
    h = pmg.Handle(1, prm)
    h.set_coefficients(pmg.coeff(kind=pmg.COEF_TABLE))
    pmg.load_hierarchy(h, levels)

    def refused(T):
        for bad in (np.nan, np.inf, -np.inf):
            for at in (0, T.size // 2, T.size - 1):
                B = 2.0 * T
                B.reshape(-1)[at] = bad
                with pytest.raises(pmg.PmgError):
                    h.set_coefficient_table(0, B)

    def table():
        T = np.random.default_rng(7).standard_normal(h.quad_points(0).shape[:2] + (6,))
        T[..., 0] = 1.0 + T[..., 0] ** 2
        return T

    T = table()
    refused(T)
    with pytest.raises(pmg.PmgError):
        h.assemble(0, fm, copy_out=False)  # still no table
    h.set_coefficient_table(0, T)
    h.assemble(0, fm, copy_out=False)
    A, b = h.get_matrix(0), h.get_rhs(0)
    refused(T)
    h.assemble(0, fm, copy_out=False)
    assert np.array_equal(h.get_matrix(0), A) and np.array_equal(h.get_rhs(0), b)
    # a table of another size, for another quadrature rule
    h.set_params(prm2 := pmg.default_params(quad_rule=getattr(pmg, "QUAD_" + other)))
    T2 = table()
    assert T2.size != T.size
    refused(T2)
    h.set_params(prm)
    h.assemble(0, fm, copy_out=False)
    assert np.array_equal(h.get_matrix(0), A) and np.array_equal(h.get_rhs(0), b)
    h.set_params(prm2)
    h.set_coefficient_table(0, T2)
    h.assemble(0, fm, copy_out=False)
    assert not np.array_equal(h.get_matrix(0), A)
    h.close()
