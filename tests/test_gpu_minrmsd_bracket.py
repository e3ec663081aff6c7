"""The bracketed minRMSD assignment against the oracle, bit for bit: frame
counts on both sides of a warp's tile and of the wide form, center counts on
both sides of a lane group, atom counts on both sides of a staged chunk, and
the inputs for which the bracket must give way to the double solve
(degenerate shapes, duplicates, coordinates far from 1, values that are not
finite)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(kind, n, n_atoms, k, rng):
    base = np.cumsum(rng.normal(size=(max(2, k // 2), n_atoms, 3)), axis=1)
    X = base[rng.integers(0, len(base), size=n)] + 0.3 * rng.normal(size=(n, n_atoms, 3))
    if kind == "planar":
        X[..., 2] = 0.0
    elif kind == "line":
        X[..., 1:] = 0.0
    elif kind == "mirror":
        X[::2, :, 0] *= -1.0
    elif kind == "tiny":
        X *= 1e-9
    elif kind == "huge":
        X *= 1e7
    X += 5.0 * rng.normal(size=(n, 1, 3)) * (0.0 if kind in ("tiny", "huge") else 1.0)
    X = X.reshape(n, 3 * n_atoms).astype(np.float32)
    C = X[rng.integers(0, n, size=k)].copy()
    if kind == "duplicate":
        C[k // 2:] = C[:k - k // 2]
    elif kind == "near":
        C = (X[rng.integers(0, n, size=1)] + 1e-4 * rng.normal(size=(k, X.shape[1]))).astype(np.float32)
    elif kind == "nan":
        X[0, 0], X[n // 2, 1], C[k - 1, 2] = np.nan, np.inf, np.nan
    return X, C


@pytest.mark.parametrize("kind,n,n_atoms,k", [
    ("plain", 1, 5, 1), ("plain", 7, 3, 31), ("plain", 9, 58, 33), ("plain", 20000, 58, 100), ("plain", 19457, 7, 65),
    ("plain", 300, 96, 40), ("plain", 300, 97, 40), ("plain", 65, 400, 10), ("plain", 40, 600, 5),
    ("plain", 500, 1, 20), ("plain", 500, 2, 20), ("planar", 1000, 12, 40), ("line", 1000, 12, 40),
    ("mirror", 1000, 20, 64), ("duplicate", 1000, 20, 64), ("near", 1000, 20, 100), ("tiny", 500, 16, 40),
    ("huge", 500, 16, 40), ("nan", 500, 16, 40)])
def test_bracketed_assignment_equals_oracle(oracle, kind, n, n_atoms, k):
    import torch
    from pyemma_gb300 import _lib as L
    X, C = _data(kind, n, n_atoms, k, np.random.default_rng(n + 31 * n_atoms + k))
    want, msd = oracle.assign_minrmsd(X, C, return_msd=True)
    lab, rmsd = L.assign_minrmsd(torch.from_numpy(X).cuda(), torch.from_numpy(C).cuda(), return_rmsd=True)
    np.testing.assert_array_equal(lab.cpu().numpy(), want)
    np.testing.assert_array_equal(rmsd.cpu().numpy(), np.sqrt(msd).astype(np.float32))
