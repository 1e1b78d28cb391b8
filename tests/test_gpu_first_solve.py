"""The set-up of a new handle's first solve: how often it allocates device memory
(one allocation above about 2 MB takes 0.3 ms whatever its size; they were what made
first solves of small hierarchies slower than with fewer tables), counted by the
profiler.  N_Q1 / Q1 24^3, four levels, FP64 SSOR.  Bar: per level one for the
copy's tables and columns, one for its values, two for what the sweeps need and three
level vectors; ten for the coarsest inverse, the Krylov vectors and the solve's own."""
import pytest

pytestmark = pytest.mark.gpu


def test_allocations_of_a_first_solve(pmg):
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.zeros(1, device="cuda")
    levels = pmg.mdml_hierarchy(pmg.Q1_HEX, 24, 3)
    counts = []
    for k in range(2):
        h = pmg.Handle(4, pmg.default_params(precision=pmg.PREC_FP64))
        h.set_coefficients(pmg.coeff(kind=pmg.COEF_CONST, eps=1e-2, b=(1, .5, .25), f=1.0))
        pmg.load_hierarchy(h, levels)
        h.assemble(-1, pmg.FORM_SUPG, copy_out=False)
        with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
            h.solve()
            torch.cuda.synchronize()
        names = [e.name for e in p.events()]
        counts.append(sum(n.startswith("cudaMalloc") for n in names))
        assert any(n.startswith("cudaGraphLaunch") for n in names)  # (the profiler does see the library's calls)
        h.close()
    assert 0 < counts[1] <= 4 * 7 + 10, counts
