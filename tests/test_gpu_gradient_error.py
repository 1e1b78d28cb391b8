"""The stencil network's backward keeps FP32 accuracy: gradients of every layer
against FP64, with everything else kept out of the comparison.

The hidden layers have one weight per output channel, a power of two, so their
pre-activations are exact and no BF16 rounding of an activation can fall the other
way; the last layer is dense; the FP64 side starts from the device's own stencil.
What differs is then the arithmetic of the backward alone: the loss gradient's
entries (5 roundings), their three BF16 parts, and the sums of data, weight and
bias gradients.

Bar: 3e-7 of each gradient's norm.  Roundings to nearest are at most 2^-24 and
sqrt(1/3) of that in the mean square; 5 of an entry and up to 40 of a sum (27 offsets
of the data gradient, runs and bricks of the weight gradient) make sqrt(45 / 3) 2^-24 =
2.3e-7 if every sum were as large as its last.  A left-out third part (2^-17 of
every entry, 2e-6) and sums that stay in the tensor cores, which round towards zero
(54 of them, 7e-7), are above it."""
import numpy as np
import pytest

from oracle import learned_oracle as LO

pytestmark = pytest.mark.gpu


def network(rng, positive):
    W1, W2 = np.zeros((32, 27, 27)), np.zeros((32, 32, 27))
    for co in range(32):
        W1[co, rng.integers(27), rng.integers(27)] = rng.choice([-1, 1]) * 2.0 ** rng.integers(-1, 2)
        W2[co, rng.integers(32), rng.integers(27)] = (1 if positive else rng.choice([-1, 1])) * 2.0 ** rng.integers(-1, 2)
    b1, b2 = LO.bf16_round(rng.uniform(0.5, 1, 32)), LO.bf16_round(rng.uniform(0.25, 0.5, 32))
    W3 = rng.uniform(0.01, 0.1, (27, 32, 27)) if positive else rng.standard_normal((27, 32, 27)) * 0.05
    b3 = LO.bf16_round(rng.standard_normal(27) * 0.05)
    return np.concatenate([x.reshape(-1) for x in (W1, b1, W2, b2, LO.bf16_round(W3), b3)]).astype(np.float32)


def gradient(theta, stencil, n1, A, Na, dof_lat, rowptr, kcol, e, r):
    """The FP64 gradients, layer by layer, for the network's activations and a given stencil."""
    f, ds = LO.features(n1, rowptr, kcol, A.data, Na, dof_lat)
    _, (f, z1, a1, z2, a2, _) = LO.forward(theta, f, ds)
    rl = LO.to_lattice(r, dof_lat, n1)
    c = LO.apply_stencil(stencil.astype(np.float64).reshape(27, n1, n1, n1), rl).reshape(-1)[dof_lat]
    c[Na:] = 0
    dc = -(A.T @ (2 * (A @ (e - c)) / float(r @ r)))
    dc[Na:] = 0
    dcl = LO.to_lattice(dc, dof_lat, n1)
    d3 = np.stack([dcl * LO.shift(rl, o) * ds for o in LO.offsets()])
    W1, b1, W2, b2, W3, b3 = LO.unpack(theta)
    da2, dW3, db3 = LO.conv_bwd(d3, a2, W3)
    dz2 = da2 * (z2 > 0)
    da1, dW2, db2 = LO.conv_bwd(dz2, a1, W2)
    _, dW1, db1 = LO.conv_bwd(da1 * (z1 > 0), f, W1)
    return [dW1.ravel(), db1, dW2.ravel(), db2, dW3.ravel(), db3]


@pytest.mark.parametrize("n,positive", [(8, False), (16, False), (21, False), (20, True)])
def test_backward_error(pmg, n, positive):
    import scipy.sparse as sp
    import scipy.sparse.linalg as sl
    import torch
    from parmoon_b200 import learned as PL
    rng = np.random.default_rng(n)
    h, lv = PL.make_problem(5, n, 1)
    F = lv[-1]
    N, Na, n1 = F["N"], F["active_bound"], n + 1
    w = network(rng, positive)
    h.set_learned_weights(w)
    A = sp.csr_matrix((h.get_matrix(0), F["kcol"], F["rowptr"]), shape=(N, N))
    stencil = h.learned_stencil(0)
    e, r = rng.standard_normal(N), rng.standard_normal(N)
    if positive:  # every sum over entries of one sign: A^T A (e - S r) < 0, r > 0
        r = rng.uniform(0.5, 1, N)
        r[Na:] = 0
        Aa = A.tocsc()[:Na, :Na]
        u = sl.spsolve(Aa, sl.spsolve(Aa.T.tocsc(), -rng.uniform(0.5, 1, Na)))
        c = LO.apply_stencil(stencil.astype(np.float64).reshape(27, n1, n1, n1), LO.to_lattice(r, F["dof_lat"], n1))
        e[:Na] = u + c.reshape(-1)[F["dof_lat"]][:Na]
    e[Na:] = r[Na:] = 0
    ed, rd = torch.from_numpy(e).cuda(), torch.from_numpy(r).cuda()
    torch.cuda.synchronize()
    _, g = h.learned_train_step(0, ed.data_ptr(), rd.data_ptr(), 1, 0.0, want_grad=True)
    h.close()
    ref = gradient(w.astype(np.float64), stencil, n1, A, Na, F["dof_lat"], F["rowptr"], F["kcol"], e, r)
    o = 0
    for name, x in zip(("W1", "b1", "W2", "b2", "W3", "b3"), ref):
        err = np.linalg.norm(g[o:o + x.size] - x) / np.linalg.norm(x)
        o += x.size
        assert err <= 3e-7, (name, err)
