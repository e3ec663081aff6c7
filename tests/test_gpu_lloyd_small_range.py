"""Lloyd runs in one cooperative launch on frames whose squared deviations are
finite in float32 but not their sums: centers and inertia stay finite and are
the oracle's (labels of a warp all equal, sorted by four lanes and by one)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k,run", [(731, 4, 2, 1), (5000, 2, 50, 1), (5000, 8, 200, 1), (1500, 1, 3, 200),
                                       (3000, 16, 20, 300)])
def test_sums_beyond_float32(oracle, n, d, k, run):
    import torch
    from pyemma_gb300 import _lib as L
    rng = np.random.default_rng(n + d)
    scale = 4.5e18 / d ** 0.5  # squared deviations of up to 1e38
    base = rng.uniform(-2, 2, size=(n // run + 1, d))
    X = (scale * (np.repeat(base, run, 0)[:n] + 0.01 * rng.normal(size=(n, d)))).astype(np.float32)
    C0 = X[rng.choice(n, size=k, replace=False)].copy()
    if run == 1:
        C0[2:] = 1e19 + 1e18 * rng.random(size=(k - 2, d))  # too far for any frame
    want = oracle.lloyd(X, C0, 1, -1.0)
    C = torch.from_numpy(C0).cuda()
    res = L.lloyd(torch.from_numpy(X).cuda(), C, 1, -1.0, precision="fp32")
    np.testing.assert_array_equal(res["labels"].cpu().numpy(), want["labels"])
    C = C.cpu().numpy()
    assert np.isfinite(C).all() and np.isfinite(res["inertias"]).all()
    np.testing.assert_allclose(C, want["centers"], rtol=0, atol=1e-6 * scale)
    np.testing.assert_allclose(res["inertias"][0], want["inertias"][0], rtol=1e-5)
