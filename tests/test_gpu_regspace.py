"""The walk of km_regspace against the oracle's frame-by-frame walk:
row widths on both sides of the register form, windows and chunks that end on
a remainder, frames that are not finite, walks in which every frame becomes a
center and walks stopped by max_centers within a window."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,dmin,max_centers", [
    (1, 3, 0.5, 10), (31, 1, 0.01, 100), (1023, 4, 0.2, 5000), (1025, 5, 0.3, 5000), (3073, 3, 0.0, 4000),
    (3073, 3, 0.0, 1500), (40000, 2, 0.01, 20000), (20000, 16, 1.0, 20000), (9000, 17, 1.2, 9000),
    (9000, 32, 1.7, 9000), (5000, 33, 1.8, 5000), (3000, 100, 3.6, 3000), (2500, 100, 3.0, 700),
    (600000, 3, 0.08, 5000)])
def test_regspace_walk_equals_oracle(oracle, n, d, dmin, max_centers):
    import torch
    from pyemma_gb300 import _lib as L
    rng = np.random.default_rng(n + d)
    X = rng.random((n, d)).astype(np.float32)
    X[n // 2:] += np.float32(0.5)  # a second region, first seen halfway
    if n > 2000 and d <= 32:
        X[7, 0] = np.nan
        X[1500, d - 1] = np.inf
        X[n - 3] = np.nan
    want, conv = oracle.regspace(X, dmin, max_centers)
    got, got_conv = L.regspace(torch.from_numpy(X).cuda(), dmin, max_centers)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    assert got_conv == conv
