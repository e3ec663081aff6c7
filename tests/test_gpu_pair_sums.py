"""Centroid sums of Lloyd runs on coordinate frames: the deviations and their
squares are rounded to float32 once each, and their sums add next to nothing to
that.  The reference rounds the same terms to float32 and sums them in float64.

Tolerance of the inertia: a compensated float32 sum of m terms is off by about
0.1 m u^2 (u = 2^-24) of its value when the roundings are independent, which is
2e-12 for the at most 4,352 squares of a lane's run of 256 rows; the runs of a
few hundred lanes and pieces average that to 1e-13.  5e-12 leaves a factor of
50.  Centers: the float32 value next to the exact one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _step(X, C, labels):
    """New centers and inertia from float32 terms summed in float64."""
    dev = X - C[labels]  # float32
    sq = dev * dev
    C2, inertia = C.copy(), 0.0
    for j in np.unique(labels):
        m = labels == j
        S, Q, cnt = dev[m].astype(np.float64).sum(0), sq[m].astype(np.float64).sum(), float(m.sum())
        mu = (C[j].astype(np.float64) + S * (1.0 / cnt)).astype(np.float32)
        dl = mu.astype(np.float64) - C[j].astype(np.float64)
        C2[j] = mu
        inertia += Q - 2.0 * (dl * S).sum() + cnt * (dl * dl).sum()
    return C2, inertia


@pytest.mark.parametrize("iters", [1, 2])  # features computed where they are read, and stored once
@pytest.mark.parametrize("prec", ["fp16", "fp32"])
@pytest.mark.parametrize("n,n_atoms,k", [(4000, 33, 20), (3001, 9, 40), (5000, 6, 7), (2500, 20, 300)])
def test_pair_sums_keep_their_bits(oracle, prec, iters, n, n_atoms, k):
    import torch
    from pyemma_gb300 import _lib as L
    rng = np.random.default_rng(n + k)
    base = np.cumsum(rng.normal(size=(8, n_atoms, 3)), axis=1)
    xyz = (base[rng.integers(0, 8, size=n)] + 0.1 * rng.normal(size=(n, n_atoms, 3))).astype(np.float32)
    xyz = torch.from_numpy(xyz).cuda()
    pairs = torch.tensor([(a, b) for a in range(n_atoms) for b in range(a + 1, n_atoms)], dtype=torch.int32).cuda()
    X = L.pair_distances(xyz, pairs).cpu().numpy()
    C = C0 = X[rng.choice(n, size=k, replace=False)].copy()
    Cd = torch.from_numpy(C0).cuda()
    r = L.lloyd_pairs(xyz, pairs, Cd, iters, -1.0, precision=prec)
    want = []
    for _ in range(iters):
        C, inertia = _step(X, C, oracle.assign(X, C))
        want.append(inertia)
    np.testing.assert_allclose(r["inertias"], want, rtol=5e-12)
    np.testing.assert_allclose(Cd.cpu().numpy(), C, rtol=2e-7, atol=0)
