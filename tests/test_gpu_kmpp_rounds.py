"""kmeans++ rounds in one launch against the oracle's draws: rows on both
sides of each register form and of the warp's form (32 features), the longest
rows, frame counts that leave partial runs and
partial groups of rows, more rounds than one launch runs, launches of one
round (with a callback), rows off the 16-byte grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prune", ["0", "1"])
@pytest.mark.parametrize("n,d,k", [
    (31, 1, 5), (33, 2, 20), (4863, 3, 70), (10007, 5, 66), (2000, 8, 65), (3001, 9, 30), (2500, 17, 40), (999, 31, 20),
    (7, 32, 7), (1001, 33, 70), (40000, 40, 129), (650, 96, 33), (300, 129, 20), (40, 4096, 9),
    (300000, 2, 10), (170000, 12, 8)])
def test_kmpp_rounds_draw_the_oracles_frames(oracle, monkeypatch, prune, n, d, k):
    import torch
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_KMPP_PRUNE", prune)
    rng = np.random.default_rng(n + d)
    X = (0.3 * rng.normal(size=(n, d)) + rng.normal(size=(9, d))[np.arange(n) * 31 // n % 9]).astype(np.float32)
    want, idx = oracle.kmpp(X, k, 77)
    flat = torch.zeros(n * d + 1, device="cuda")
    for shift in (0, 1):
        Xd = flat[shift:shift + n * d].view(n, d)
        Xd.copy_(torch.from_numpy(X))
        for callback in (None, lambda: None):
            C, got = L.kmpp(Xd, k, 77, callback=callback)
            np.testing.assert_array_equal(got.cpu().numpy(), idx)
            np.testing.assert_array_equal(C.cpu().numpy(), want)


@pytest.mark.parametrize("prune", ["0", "1"])
def test_kmpp_rounds_take_what_is_not_finite(oracle, monkeypatch, prune):
    import torch
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_KMPP_PRUNE", prune)
    for d in (3, 40):
        X = np.random.default_rng(d).normal(size=(3000, d)).astype(np.float32)
        X[5, 1], X[600, 0], X[601], X[2999, 2] = np.nan, np.inf, 3e38, -np.inf
        want, idx = oracle.kmpp(X, 12, 3)
        C, got = L.kmpp(torch.from_numpy(X).cuda(), 12, 3)
        np.testing.assert_array_equal(got.cpu().numpy(), idx)
        np.testing.assert_array_equal(C.cpu().numpy(), want)
