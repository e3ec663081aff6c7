"""The narrow-frame assignment (split FP16 operands, exact distances of the
best eight centers) against the oracle, label for label: feature counts on
both sides of a K step and of an operand panel, frame counts on both sides of
a tile, center counts on both sides of a group, a column tile and the sets
that one launch keeps in shared memory, and inputs that send frames to the
re-check over all centers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _labels(L, X, C, precision="fp16"):
    import torch
    lab, stats = L.assign(torch.from_numpy(X).cuda(), torch.from_numpy(C).cuda(), precision=precision)
    return lab.cpu().numpy(), stats


@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 7, 8, 11, 12, 15, 16, 19, 20, 31])
@pytest.mark.parametrize("n,k", [(1, 1), (127, 7), (128, 8), (129, 9), (1000, 127), (5000, 129), (40001, 512),
                                 (3000, 1153), (2000, 2500)])
def test_small_equals_oracle(oracle, monkeypatch, d, n, k):
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_TC_SMALL", "1")
    rng = np.random.default_rng(100 * d + n + k)
    X = (rng.normal(size=(n, d)) + 3.0 * rng.integers(0, 3, size=(n, 1))).astype(np.float32)
    C = (X[rng.integers(0, n, size=k)] + 0.05 * rng.normal(size=(k, d))).astype(np.float32)
    want = oracle.assign(X, C)
    for precision in ("fp16", "auto"):
        got, _ = _labels(L, X, C, precision)
        np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("kind", ["duplicate", "lattice", "offset", "outlier", "nonfinite", "same", "scale"])
@pytest.mark.parametrize("d", [2, 10, 20])
def test_small_hard_inputs(oracle, monkeypatch, kind, d):
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_TC_SMALL", "1")
    rng = np.random.default_rng(d)
    n, k = 3000, 300
    X = rng.normal(size=(n, d)).astype(np.float32)
    C = X[rng.integers(0, n, size=k)].copy()
    if kind == "duplicate":
        C[k // 2:] = C[:k - k // 2]
    elif kind == "lattice":
        X, C = np.round(X), np.round(2 * C) / 2
    elif kind == "offset":
        X, C = X * 1e-2 + 1e4, C * 1e-2 + 1e4
    elif kind == "outlier":
        X[::50] *= 1e5
        X[7] *= 1e18
    elif kind == "nonfinite":
        X[5, 0], X[6, d - 1], X[7, :] = np.nan, np.inf, -np.inf
        C[11, 0] = np.nan
    elif kind == "same":
        C[:] = C[0]
    elif kind == "scale":
        X, C = X * 1e-12, C * 1e-12
    X, C = X.astype(np.float32), C.astype(np.float32)
    got, stats = _labels(L, X, C)
    np.testing.assert_array_equal(got, oracle.assign(X, C))
    if kind in ("duplicate", "same"):
        assert stats["n_full"] > 0


@pytest.mark.parametrize("n,d,k", [(70001, 3, 100), (50000, 10, 1000), (30000, 24, 700)])
def test_small_lloyd_and_resident_equal_plain(monkeypatch, n, d, k):
    import torch
    from pyemma_gb300 import _lib as L
    rng = np.random.default_rng(n)
    X = torch.from_numpy(rng.normal(size=(n, d)).astype(np.float32)).cuda()
    C0 = X[torch.from_numpy(rng.choice(n, k, replace=False)).cuda()].contiguous()
    out = {}
    for form in ("0", "1"):
        monkeypatch.setenv("KM_TC_SMALL", form)
        C = C0.clone()
        r = L.lloyd(X, C, 4, -1.0, precision="fp16")
        P = C0.clone()
        h = L.lloyd_host([X.cpu().numpy()], P, 1, -1.0, precision="fp16")
        lab, _ = L.Centers(C0, precision="fp16").assign(X)
        out[form] = (r["labels"], C, r["inertias"], lab, h["labels"])
    assert torch.equal(out["0"][3], out["1"][3])
    assert torch.equal(out["0"][4], out["1"][4])
    assert (out["0"][0] != out["1"][0]).sum().item() <= 3  # float64 sums in another order
    torch.testing.assert_close(out["0"][1], out["1"][1], rtol=1e-4, atol=1e-5)
    np.testing.assert_allclose(out["0"][2], out["1"][2], rtol=1e-6)
