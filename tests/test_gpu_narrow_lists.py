"""Narrow frames that the first pass cannot settle: labels against the exact
kernel on both sides of the list length (32,768) and of the work (2e10) from
which eight frames share a warp and a second pass is made, with exact ties,
lattice data, frames and centers that are not finite, one and several launches
over the centers, lists longer than the room for the bits, and inside Lloyd
runs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frames(kind, n, d, k, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    X = torch.randn((n, d), generator=g, device="cuda")
    C = X[torch.randint(0, n, (k,), generator=g, device="cuda")].clone()
    if kind in ("twice", "mixed"):
        C[k // 2:2 * (k // 2)] = C[:k // 2].clone()
    if kind == "lattice":
        X, C = torch.round(2 * X) / 2, torch.round(2 * C) / 2
    if kind == "mixed":  # frames without a bound among those with one
        X[::3, 0] = float("nan")
        X[1::97] = float("inf")
        X[5::101] *= 1e19
    if kind == "nan_center":
        C[k // 3, 0] = float("nan")
    return X.contiguous(), C.contiguous()


@pytest.mark.parametrize("kind", ["twice", "lattice", "mixed", "nan_center"])
@pytest.mark.parametrize("n,d,k", [
    (32768, 3, 64000), (32769, 3, 64000), (32775, 15, 14000), (40001, 2, 4000), (200_003, 10, 4000),
    (300_011, 24, 1000), (150_007, 31, 1500), (50003, 1, 9000), (250_001, 16, 2048), (33001, 4, 129), (40005, 10, 1000)])
def test_long_lists_equal_exact(monkeypatch, kind, n, d, k):
    import torch
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_TC_SMALL", "1")
    X, C = _frames(kind, n, d, k, n + d)
    want = L.assign(X, C, precision="fp32")[0]
    for prec in ("fp16", "auto"):
        got, stats = L.assign(X, C, precision=prec)
        assert torch.equal(got, want)
        got, stats = L.Centers(C, precision=prec).assign(X)
        assert torch.equal(got, want)
    if kind in ("twice", "nan_center"):
        assert stats["n_full"] >= n - n // 50


def test_more_frames_than_room_for_bits():
    import torch
    from pyemma_gb300 import _lib as L
    n, d, k = 3_400_000, 2, 5000  # room for 3,195,660
    X, C = _frames("twice", n, d, k, 1)
    got, stats = L.assign(X, C, precision="fp16")
    assert stats["n_full"] > 3_300_000
    assert torch.equal(got, L.assign(X, C, precision="fp32")[0])


@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("kind,n,d,k", [("lattice", 2_600_000, 2, 1000), ("lattice", 200_000, 2, 500), ("twice", 100_000, 6, 900),
                                        ("twice", 60_000, 24, 600), ("plain", 100_000, 5, 700)])
def test_lloyd_settles_long_lists(oracle, monkeypatch, host, kind, n, d, k):
    import torch
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_TC_SMALL", "1")
    X, C0 = _frames(kind, n, d, k, n)
    Xh, entering = X.cpu().numpy(), [C0.cpu().numpy()]
    C = C0.clone()
    progress = lambda: entering.append(C.cpu().numpy())
    if host:
        r = L.lloyd_host([Xh[:n // 3], Xh[n // 3:]], C, 3, -1.0, callback=progress)
    else:
        r = L.lloyd(X, C, 3, -1.0, callback=progress)
    np.testing.assert_array_equal(r["labels"].cpu().numpy(), oracle.assign(Xh, entering[2]))
    P = C0.clone()
    L.lloyd(X, P, 3, -1.0)  # the iterations as one device-side loop
    torch.testing.assert_close(P, C, rtol=1e-4, atol=1e-5)
