"""Lloyd runs whose tensor-core passes leave out center tiles by the triangle
inequality, against the runs that compare every frame with every center: the
labels and counts are the same, including ties (duplicate frames and centers),
units of frames that change clusters, ragged last units, centers that end a
partial tile, both tile forms, and frames that are not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _runs(monkeypatch, X, C0, iters, prec, **env):
    import torch
    from pyemma_gb300 import _lib as L
    out = []
    for bounds in ("0", "1"):
        monkeypatch.setenv("KM_TC_BOUNDS", bounds)
        for key, v in env.items():
            monkeypatch.setenv(key, v)
        C = torch.from_numpy(C0).cuda()
        r = L.lloyd(torch.from_numpy(X).cuda(), C, iters, -1.0, precision=prec)
        out.append((r["labels"].cpu().numpy(), C.cpu().numpy(), np.asarray(r["inertias"])))
    return out


def _dwelling(n, d, states, rng, spread=4.0, jitter=0.3):
    means = spread * rng.normal(size=(states, d))
    which = np.repeat(rng.integers(0, states, size=n // 150 + 1), 150)[:n]
    return (means[which] + jitter * rng.normal(size=(n, d))).astype(np.float32)


@pytest.mark.parametrize("pair", ["0", "1"])
@pytest.mark.parametrize("prec,n,d,k", [
    ("fp16", 20000, 64, 600), ("fp16", 10001, 130, 1025), ("bf16", 9999, 96, 520), ("fp16", 300, 40, 290),
    ("fp16", 70001, 33, 2100), ("fp16", 12000, 700, 300), ("fp16", 4000, 32, 4000)])
def test_bounded_lloyd_equals_full(oracle, monkeypatch, pair, prec, n, d, k):
    rng = np.random.default_rng(n + k)
    X = _dwelling(n, d, 40, rng)
    X[n // 3:n // 3 + 200] = X[5]  # ties
    C0 = X[rng.choice(n, size=k, replace=False)].copy()
    C0[1] = C0[0]
    (la, Ca, ia), (lb, Cb, ib) = _runs(monkeypatch, X, C0, 4, prec, KM_TC_PAIR=pair)
    np.testing.assert_allclose(Cb, Ca, rtol=1e-5, atol=1e-5)
    np.testing.assert_allclose(ib, ia, rtol=1e-6)
    assert (la != lb).sum() <= 2  # float64 sums in another order
    (la, _, _), (lb, _, _) = _runs(monkeypatch, X, C0, 2, prec, KM_TC_PAIR=pair)
    want = oracle.lloyd(X, C0, 2, -1.0)["labels"]
    assert (lb != want).sum() <= 2 and (la != want).sum() <= 2


def test_bounded_lloyd_takes_what_is_not_finite(monkeypatch):
    rng = np.random.default_rng(3)
    X = _dwelling(6000, 64, 20, rng)
    X[7, 3], X[3000, 0] = np.nan, np.inf
    C0 = X[rng.choice(2900, size=300, replace=False) + 8].copy()
    (la, Ca, _), (lb, Cb, _) = _runs(monkeypatch, X, C0, 3, "fp16")
    np.testing.assert_array_equal(np.isfinite(Ca), np.isfinite(Cb))
    assert (la != lb).sum() <= 2
