"""Center bounds and the narrow-frame kernel: FP16 Lloyd runs on narrow frames
keep no bounds (that kernel neither writes nor reads them), reserve no room for
them, and give the same with the bounds forced on; a workspace without the room
that the bounds would take runs without them."""
import ctypes

import numpy as np
import pytest


def test_narrow_lloyd_reserves_no_bounds(kmlib, monkeypatch):
    n, d, k, fp16 = 5_000_000, 24, 2000, 1
    monkeypatch.setenv("KM_TC_SMALL", "0")
    general = kmlib.km_lloyd_workspace_size(n, d, k, fp16)
    monkeypatch.setenv("KM_TC_SMALL", "1")
    assert kmlib.km_lloyd_workspace_size(n, d, k, fp16) <= general - 4 * n


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,k", [(20000, 24, 700), (9001, 31, 600), (15000, 10, 1025)])
def test_narrow_lloyd_with_bounds_forced(oracle, monkeypatch, n, d, k):
    import torch
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_TC_BOUNDS", "1")
    rng = np.random.default_rng(n)
    X = (np.repeat(rng.normal(size=(n // 100 + 1, d)), 100, axis=0)[:n] + 0.2 * rng.normal(size=(n, d)))
    X = X.astype(np.float32)
    C0 = X[rng.choice(n, size=k, replace=False)].copy()
    Xd = torch.from_numpy(X).cuda()
    entering = [C0]
    C = torch.from_numpy(C0).cuda()
    r = L.lloyd(Xd, C, 4, -1.0, precision="fp16", callback=lambda: entering.append(C.cpu().numpy()))
    np.testing.assert_array_equal(r["labels"].cpu().numpy(), oracle.assign(X, entering[3]))
    C = torch.from_numpy(C0).cuda()
    L.lloyd(Xd, C, 4, -1.0, precision="fp16")  # the iterations as one device-side loop
    np.testing.assert_allclose(C.cpu().numpy(), entering[4], rtol=1e-4, atol=1e-5)


@pytest.mark.gpu
def test_bounds_need_their_room(oracle, monkeypatch):
    import torch
    from pyemma_gb300 import _lib as L
    lib = L.load()
    monkeypatch.setenv("KM_TC_BOUNDS", "1")
    n, d, k, p = 8000, 64, 600, L.precision_code("fp16")
    rng = np.random.default_rng(1)
    X = rng.normal(size=(n, d)).astype(np.float32)
    C0 = X[:k].copy()
    Xd = torch.from_numpy(X).cuda()
    size = lib.km_lloyd_workspace_size(n, d, k, p)
    want = oracle.lloyd(X, C0, 3, -1.0)
    for room in (size, size - 4 * n):
        ws = torch.full((size,), 7, dtype=torch.uint8, device="cuda")
        C, labels = torch.from_numpy(C0).cuda(), torch.empty(n, dtype=torch.int32, device="cuda")
        it, conv = ctypes.c_int32(0), ctypes.c_int32(0)
        L.check(lib.km_lloyd(L._ptr(Xd), n, d, k, L._ptr(C), 3, -1.0, p, L._ptr(labels), None, ctypes.byref(it),
                             ctypes.byref(conv), L._callback(None)[0], None, L._ptr(ws), room,
                             L._stream(torch, Xd.device)))
        assert bool((ws[room:] == 7).all())
        np.testing.assert_allclose(C.cpu().numpy(), want["centers"], rtol=1e-5, atol=1e-5)
