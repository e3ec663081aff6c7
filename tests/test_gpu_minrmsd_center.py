"""Centering of minRMSD frames on both sides of the frame and atom counts from
which a thread takes a row (19,456 rows of up to 128 atoms, 77,824 of up to 150;
a warp per row below and for longer rows): labels and distances of the oracle,
bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,n_atoms,k", [
    (19455, 128, 3), (19456, 128, 3), (19456, 129, 3), (77823, 150, 2), (77824, 129, 2), (77824, 150, 2),
    (77824, 151, 2)])
def test_centering_equals_oracle(oracle, n, n_atoms, k):
    import torch
    from pyemma_gb300 import _lib as L
    rng = np.random.default_rng(n + n_atoms)
    base = np.cumsum(rng.normal(size=(8, n_atoms, 3)), axis=1)
    X = base[rng.integers(0, 8, size=n)] + 0.3 * rng.normal(size=(n, n_atoms, 3)) + 5.0 * rng.normal(size=(n, 1, 3))
    X = X.reshape(n, -1).astype(np.float32)
    X[7] *= 1e-20  # beside a row whose values span many bits
    X[8, ::5] *= 1e-12
    C = X[rng.integers(0, n, size=k)].copy()
    want, msd = oracle.assign_minrmsd(X, C, return_msd=True)
    lab, rmsd = L.assign_minrmsd(torch.from_numpy(X).cuda(), torch.from_numpy(C).cuda(), return_rmsd=True)
    np.testing.assert_array_equal(lab.cpu().numpy(), want)
    np.testing.assert_array_equal(rmsd.cpu().numpy(), np.sqrt(msd).astype(np.float32))
