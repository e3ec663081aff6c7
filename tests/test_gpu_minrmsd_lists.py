"""minRMSD assignment with more centers without a bracket than a frame's list
holds (many centers, flat or two-sided structures), with crowds of near-ties
that come at once, and on both sides of the frame count (eight per SM), the
center count (32) and the atom counts (192, 384) from which frames are
bracketed: labels and distances of the oracle, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,n_atoms,k", [
    ("plain", 1500, 10, 1000), ("plain", 1501, 5, 3000), ("flat", 1300, 12, 700), ("mirror", 1400, 20, 900),
    ("crowd", 1300, 20, 600), ("crowd", 1300, 9, 33), ("plain", 1216, 9, 32), ("plain", 1217, 9, 32),
    ("plain", 1216, 9, 33), ("plain", 40, 192, 40), ("plain", 40, 191, 40), ("plain", 1300, 200, 40),
    ("plain", 2432, 384, 5), ("plain", 2433, 384, 5),
    ("plain", 2433, 383, 5), ("flat", 3, 12, 700), ("nan", 1300, 16, 500)])
def test_long_lists_equal_oracle(oracle, kind, n, n_atoms, k):
    import torch
    from pyemma_gb300 import _lib as L
    rng = np.random.default_rng(n + 31 * n_atoms + k)
    base = np.cumsum(rng.normal(size=(40, n_atoms, 3)), axis=1)
    X = base[rng.integers(0, 40, size=n)] + 0.3 * rng.normal(size=(n, n_atoms, 3))
    C = base[rng.integers(0, 40, size=k)] + 0.3 * rng.normal(size=(k, n_atoms, 3))
    if kind == "flat":
        X[..., 2], C[..., 2] = 0.0, 0.0
    elif kind == "mirror":
        C[::2, :, 0] *= -1.0
    elif kind == "crowd":  # runs of equal centers among others
        C[40:75] = C[3]
        C[k // 2:k // 2 + 9] = C[k // 3] + 1e-7 * rng.normal(size=(n_atoms, 3))
    X, C = X.reshape(n, -1).astype(np.float32), C.reshape(k, -1).astype(np.float32)
    if kind == "nan":
        X[0, 0], X[n // 2, 1], C[k - 1, 2], C[5, 0] = np.nan, np.inf, np.nan, np.inf
    want, msd = oracle.assign_minrmsd(X, C, return_msd=True)
    lab, rmsd = L.assign_minrmsd(torch.from_numpy(X).cuda(), torch.from_numpy(C).cuda(), return_rmsd=True)
    np.testing.assert_array_equal(lab.cpu().numpy(), want)
    np.testing.assert_array_equal(rmsd.cpu().numpy(), np.sqrt(msd).astype(np.float32))
