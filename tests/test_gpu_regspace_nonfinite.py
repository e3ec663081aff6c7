"""Regular space walks of wide rows (d > 32) over several chunks with frames
that are not finite: a distance that is NaN is not at least dmin, whichever
chunk its center comes from."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["first", "inf", "mixed", "overflow"])
@pytest.mark.parametrize("n,d", [(1025, 33), (5706, 33), (2100, 100), (70000, 40)])
def test_wide_walk_with_nonfinite_frames(oracle, kind, n, d):
    import torch
    from pyemma_gb300 import _lib as L
    rng = np.random.default_rng(n + d)
    X = rng.random((n, d)).astype(np.float32)
    dmin = 0.45 * d ** 0.5
    if kind == "first":  # a center that no other frame is away from
        X[0, d - 1] = np.nan
    elif kind == "inf":  # equal signs: NaN distances between such frames, others infinite
        X[::37, 4] = np.inf
        X[11::53, d - 2] = -np.inf
    elif kind == "mixed":
        X[5::41, 0] = np.nan
        X[7::29, 3] = np.inf
        X[n - 1] = np.inf
    else:  # finite, with distances that overflow
        X[3::19] *= np.float32(1e30)
    want, conv = oracle.regspace(X, dmin, 3000)
    got, got_conv = L.regspace(torch.from_numpy(X).cuda(), dmin, 3000)
    np.testing.assert_array_equal(got.cpu().numpy(), want)
    assert got_conv == conv
