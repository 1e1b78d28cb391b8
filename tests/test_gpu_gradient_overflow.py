"""A gradient that overflows FP32 at one node stays what FP32 arithmetic makes of
it: infinite, not NaN.  The loss gradient is infinite at the middle node of the
lattice alone (e is one large value there, and A^T A e is within FP32 elsewhere);
with positive activations and positive weights behind it every sum of the last
layer's and the second layer's weight and bias gradients takes that infinity in
with factors that are not 0, and no other infinity."""
import numpy as np
import pytest

from oracle import learned_oracle as LO
from test_gpu_gradient_error import network

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_infinite_not_nan(pmg, sign):
    import scipy.sparse as sp
    import torch
    from parmoon_b200 import learned as PL
    n, n1 = 8, 9
    h, lv = PL.make_problem(5, n, 1)
    F = lv[-1]
    N, Na = F["N"], F["active_bound"]
    a = h.get_matrix(0)
    rows = np.repeat(np.arange(N), np.diff(F["rowptr"]))
    act = rows < Na
    a[act] *= 2.0 ** np.round(np.log2(64.0 / np.median(a[(F["kcol"] == rows) & act])))  # diagonal about 64
    h.set_matrix(0, a)
    # first layer: the tap on the diagonal's feature (1 at active nodes) or none, so activations are > 0 everywhere
    rng = np.random.default_rng(1)
    w = network(rng, True)
    W1 = np.zeros((32, 27, 27), dtype=np.float32)
    W1[:, 13, 13] = 0.5
    w[:W1.size] = W1.reshape(-1)
    h.set_learned_weights(w)
    A = sp.csr_matrix((a, F["kcol"], F["rowptr"]), shape=(N, N))
    mid = int(np.flatnonzero(F["dof_lat"] == 4 + n1 * (4 + n1 * 4))[0])
    e, r = np.zeros(N), np.ones(N)
    e[mid] = 1.0
    # the middle value of A^T A e to 1.3 x 2^128, the others below 0.95 x 2^128
    du = A.T @ (A @ e)
    dv = np.abs(du) / du[mid]
    assert 1.3 * np.sort(dv)[-2] < 0.95
    e *= sign * 1.3 * 2.0 ** 128 / du[mid]
    ed, rd = torch.from_numpy(e).cuda(), torch.from_numpy(r).cuda()
    torch.cuda.synchronize()
    _, g = h.learned_train_step(0, ed.data_ptr(), rd.data_ptr(), 1, 0.0, want_grad=True)
    h.close()
    o = np.cumsum([0] + LO.SIZES)
    for name, k in (("b3", 5), ("W3", 4), ("b2", 3), ("W2", 2)):
        x = g[o[k]:o[k + 1]]
        assert np.all(np.isinf(x)), (name, np.isnan(x).sum(), np.isinf(x).sum(), x.size)
        assert np.all(np.sign(x) == np.sign(x[0])), name
