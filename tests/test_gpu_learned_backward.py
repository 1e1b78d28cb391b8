"""The network's gradient on the tensor cores (three BF16 parts of every FP32
gradient) against the FP64 oracle, on lattices that cut the bricks in every way:
8^3 nodes (half a brick), 16^3 (whole bricks), 17^3 and 21^3 (one node over, and
odd), one and two samples.  Bars as test_gpu_learned.py derives them: loss and
gradient within 1e-3 (the forward's BF16 roundings); two calls agree bitwise."""
import numpy as np
import pytest

from oracle import learned_oracle as LO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,samples", [(7, 1), (15, 2), (16, 1), (20, 2)])
def test_gradient_matches_oracle(pmg, n, samples):
    import torch
    from parmoon_b200 import learned as PL
    # a coarsest level of at most 832 active rows is not needed here: no solve
    h, lv = PL.make_problem(5, n, 1)
    F = lv[-1]
    N, Na = F["N"], F["active_bound"]
    rng = np.random.default_rng(n)
    w = (rng.standard_normal(LO.n_params()) * 0.05).astype(np.float32)
    h.set_learned_weights(w)
    A = h.get_matrix(0)
    E = rng.standard_normal((samples, N))
    E[:, Na:] = 0
    R = np.stack([h.matvec(0, e) for e in E])
    R[:, Na:] = 0
    Ed, Rd = torch.from_numpy(E).cuda(), torch.from_numpy(R).cuda()
    loss, g = h.learned_train_step(0, Ed.data_ptr(), Rd.data_ptr(), samples, 0.0, want_grad=True)
    loss2, g2 = h.learned_train_step(0, Ed.data_ptr(), Rd.data_ptr(), samples, 0.0, want_grad=True)
    assert loss == loss2 and np.array_equal(g, g2)
    ref = [LO.loss_and_grad(LO.bf16_round(w), n + 1, F["rowptr"], F["kcol"], A, Na, F["dof_lat"], e, r)
           for e, r in zip(E, R)]
    lo, go = np.mean([r[0] for r in ref]), np.mean([r[1] for r in ref], axis=0)
    assert abs(loss - lo) <= 1e-3 * lo, abs(loss - lo) / lo
    assert np.linalg.norm(g - go) <= 1e-3 * np.linalg.norm(go), np.linalg.norm(g - go) / np.linalg.norm(go)
    h.close()
