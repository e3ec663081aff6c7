"""Frames with more possible centers than a candidate list holds, taken a
second time by the tensor-core pass: labels against the oracle, for crowded
centers (many within the rounding bound), exact ties, both list lengths and
tile forms, partial center tiles, more such frames than there is room for
copies, short lists that keep the full re-check, frames that are not finite,
and inside Lloyd runs and their chunks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _crowded(n, d, k, groups, rng, tight):
    means = 5.0 * rng.normal(size=(groups, d))
    C = means[rng.integers(0, groups, size=k)] + tight * rng.normal(size=(k, d))
    X = means[rng.integers(0, groups, size=n)] + 0.2 * rng.normal(size=(n, d))
    return X.astype(np.float32), C.astype(np.float32)


@pytest.mark.parametrize("pair", ["0", "1"])
@pytest.mark.parametrize("prec,n,d,k,groups,tight", [
    ("fp16", 20000, 64, 600, 4, 1e-4), ("fp16", 9001, 300, 1025, 20, 1e-3), ("bf16", 8000, 96, 520, 8, 1e-2),
    ("fp16", 5000, 40, 100, 3, 1e-4), ("fp16", 30000, 33, 290, 280, 1e-3), ("fp16", 6000, 700, 300, 6, 1e-3)])
def test_crowded_lists_equal_oracle(oracle, monkeypatch, pair, prec, n, d, k, groups, tight):
    import torch
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_TC_PAIR", pair)
    rng = np.random.default_rng(n + k)
    X, C = _crowded(n, d, k, groups, rng, tight)
    C[k // 2:k // 2 + 20] = C[3]  # ties
    X[11, 2], X[n - 1, 0] = np.nan, np.inf
    want = oracle.assign(X, C)
    Xd, Cd = torch.from_numpy(X).cuda(), torch.from_numpy(C).cuda()
    full = {}
    for wide in ("0", "1"):
        monkeypatch.setenv("KM_TC_WIDE", wide)
        lab, stats = L.assign(Xd, Cd, precision=prec)
        np.testing.assert_array_equal(lab.cpu().numpy(), want)
        full[wide] = stats["n_full"]
    assert full["0"] == full["1"] > 0


def test_crowded_lists_in_lloyd(monkeypatch):
    import torch
    from pyemma_gb300 import _lib as L
    rng = np.random.default_rng(8)
    X, C0 = _crowded(600000, 32, 400, 300, rng, 0.05)  # two chunks
    X[::7] = X[0]
    C0[:50] = X[0] + 1e-5 * rng.normal(size=(50, 32)).astype(np.float32)
    out = []
    for wide in ("0", "1"):
        monkeypatch.setenv("KM_TC_WIDE", wide)
        for bounds in ("0", "1"):
            monkeypatch.setenv("KM_TC_BOUNDS", bounds)
            C = torch.from_numpy(C0).cuda()
            r = L.lloyd(torch.from_numpy(X).cuda(), C, 3, -1.0, precision="fp16")
            out.append((r["labels"].cpu().numpy(), C.cpu().numpy()))
    for lab, C in out[1:]:
        assert (lab != out[0][0]).sum() <= 2  # float64 sums in another order
        np.testing.assert_allclose(C, out[0][1], rtol=1e-5, atol=1e-5)
