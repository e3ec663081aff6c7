"""Lloyd runs of few, narrow centers in one launch against the oracle: frame
counts on both sides of a CTA and of the resident CTAs, register forms of the
features, center counts up to the shared-memory limit, more iterations than
one launch runs, clusters that empty, one label for every frame, callbacks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(X, C0, max_iter, tol, **kw):
    import torch
    from pyemma_gb300 import _lib as L
    C = torch.from_numpy(C0).cuda()
    r = L.lloyd(torch.from_numpy(X).cuda(), C, max_iter, tol, precision="fp32", **kw)
    return r, C.cpu().numpy()


@pytest.mark.parametrize("n,d,k,iters", [
    (1, 1, 1, 3), (511, 2, 7, 5), (513, 3, 40, 5), (4097, 4, 1, 4), (20000, 5, 33, 6), (20000, 8, 60, 6),
    (30000, 9, 50, 5), (30000, 16, 200, 5), (100000, 2, 50, 70), (700001, 1, 12, 130), (200000, 2, 900, 4)])
def test_small_lloyd_equals_oracle(oracle, n, d, k, iters):
    rng = np.random.default_rng(n + d + k)
    X = (rng.normal(size=(n, d)) + 4.0 * rng.integers(0, 4, size=(n, 1))).astype(np.float32)
    C0 = X[rng.integers(0, n, size=k)] + np.float32(0.01) * rng.normal(size=(k, d)).astype(np.float32)
    got, C = _run(X, C0, iters, -1.0)
    want = oracle.lloyd(X, C0, iters, -1.0)
    assert got["n_iter"] == want["n_iter"] == iters
    np.testing.assert_allclose(C, want["centers"], rtol=1e-5, atol=1e-5)
    np.testing.assert_allclose(got["inertias"], want["inertias"], rtol=1e-6)
    assert (got["labels"].cpu().numpy() != want["labels"]).sum() <= 2  # float64 sums in another order


def test_small_lloyd_stops_empties_and_calls_back(oracle):
    rng = np.random.default_rng(4)
    X = rng.normal(size=(5000, 2)).astype(np.float32)
    C0 = np.concatenate([X[:6], 100 + X[:3]]).astype(np.float32)  # three clusters without members
    calls = []
    for cb in (None, lambda: calls.append(1)):
        got, C = _run(X, C0, 100, 1e-5, callback=cb)
        want = oracle.lloyd(X, C0, 100, 1e-5)
        assert got["converged"] and want["converged"] and got["n_iter"] == want["n_iter"]
        np.testing.assert_allclose(C, want["centers"], rtol=1e-5, atol=1e-5)
        np.testing.assert_array_equal(C[6:], C0[6:])
    assert len(calls) == got["n_iter"]
    same = np.tile(X[:1], (4000, 1))  # every frame in one cluster, inertia 0
    got, C = _run(same, X[:4].copy(), 5, -1.0)
    want = oracle.lloyd(same, X[:4].copy(), 5, -1.0)
    np.testing.assert_array_equal(got["labels"].cpu().numpy(), want["labels"])
    np.testing.assert_allclose(C, want["centers"], rtol=1e-6)
