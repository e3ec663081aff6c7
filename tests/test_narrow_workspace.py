"""Workspaces of narrow frames under "auto": a few bytes per frame for the
lists of the narrow-frame kernel, none for Lloyd runs that go in one
cooperative launch, and calls with only the exact kernel's workspace still run,
with the same labels, without a byte written beyond what they were given."""
import ctypes

import numpy as np
import pytest

FP32, FP16, AUTO = 0, 1, 2


@pytest.mark.parametrize("n,d,k", [(10_000_000, 2, 500), (4_000_000, 3, 200), (100_000_000, 7, 900)])
def test_lists_take_four_bytes_per_frame(kmlib, n, d, k):
    fixed = (256 + 8) << 20  # a second pass's bits, the centers' operands
    assert 4 * n <= kmlib.km_assign_workspace_size(n, d, k, AUTO) <= 4 * n + fixed
    plain = kmlib.km_lloyd_workspace_size(n, d, k, FP32)
    assert kmlib.km_lloyd_workspace_size(n, d, k, AUTO) <= plain + 16 * n + fixed


def test_more_centers_than_a_launch_holds(kmlib):
    n, d, k = 10_000_000, 24, 900
    assert kmlib.km_assign_workspace_size(n, d, k, AUTO) <= 16 * n + (264 << 20)


def test_cooperative_lloyd_takes_no_lists(kmlib):
    for n, d, k in ((1_000_000, 2, 200), (4_000_000, 6, 50)):
        assert kmlib.km_assign_workspace_size(n, d, k, AUTO) > 0  # its assignment alone is narrow
        assert kmlib.km_lloyd_workspace_size(n, d, k, AUTO) == kmlib.km_lloyd_workspace_size(n, d, k, FP32)


def _lloyd(L, X, C0, p, size):
    import torch
    lib = L.load()
    n, d = X.shape
    ws = torch.full((size + 64,), 7, dtype=torch.uint8, device="cuda")
    C, labels = C0.clone(), torch.empty(n, dtype=torch.int32, device="cuda")
    it, conv = ctypes.c_int32(0), ctypes.c_int32(0)
    L.check(lib.km_lloyd(L._ptr(X), n, d, len(C0), L._ptr(C), 3, -1.0, p, L._ptr(labels), None, ctypes.byref(it),
                         ctypes.byref(conv), L._callback(None)[0], None, L._ptr(ws), size,
                         L._stream(torch, X.device)))
    assert bool((ws[size:] == 7).all())
    return C.cpu().numpy(), labels.cpu().numpy()


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,k", [(1, 4, 3), (200_001, 5, 500), (60_000, 3, 1500), (30_000, 24, 700)])
def test_narrow_calls_in_the_exact_kernels_workspace(oracle, monkeypatch, n, d, k):
    import torch
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_TC_SMALL", "1")
    lib = L.load()
    rng = np.random.default_rng(n)
    Xh = rng.normal(size=(n, d)).astype(np.float32)
    Ch = (Xh[rng.integers(0, n, size=k)] + 0.01 * rng.normal(size=(k, d))).astype(np.float32)
    want = oracle.assign(Xh, Ch)
    X, C = torch.from_numpy(Xh).cuda(), torch.from_numpy(Ch).cuda()
    h = L.Centers(C)
    s = L._stream(torch, X.device)
    sizes = [lib.km_assign_workspace_size(n, d, k, AUTO), lib.km_assign_centers_workspace_size(n, h.handle)]
    assert min(sizes) >= 4 * n
    for full, resident in zip(sizes, (False, True)):
        for size in (full, 4 * n - 4, 0):
            ws = torch.full((size + 64,), 7, dtype=torch.uint8, device="cuda")
            lab = torch.full((n,), -1, dtype=torch.int32, device="cuda")
            st = L.AssignStats()
            ptr = L._ptr(ws) if size else None
            if resident:
                L.check(lib.km_assign_centers(L._ptr(X), n, d, h.handle, L._ptr(lab), ptr, size, ctypes.byref(st), s))
            else:
                L.check(lib.km_assign(L._ptr(X), n, d, L._ptr(C), k, AUTO, L._ptr(lab), ptr, size, ctypes.byref(st),
                                      s))
            np.testing.assert_array_equal(lab.cpu().numpy(), want)
            assert bool((ws[size:] == 7).all())
    ends = [_lloyd(L, X, C, AUTO, lib.km_lloyd_workspace_size(n, d, k, p)) for p in (AUTO, FP32)]
    np.testing.assert_allclose(ends[1][0], ends[0][0], rtol=1e-4, atol=1e-5)


@pytest.mark.gpu
def test_no_memory_for_the_lists(oracle, monkeypatch):
    import torch
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_TC_SMALL", "1")
    rng = np.random.default_rng(0)
    Xh = rng.normal(size=(5000, 3)).astype(np.float32)
    Ch = Xh[:100].copy()
    X, C = torch.from_numpy(Xh).cuda(), torch.from_numpy(Ch).cuda()
    h = L.Centers(C)
    plain = L.load().km_lloyd_workspace_size(5000, 3, 100, FP32)
    room = L._workspace

    def short(torch_, nbytes, device):
        if nbytes > plain:
            raise torch.OutOfMemoryError("none left")
        return room(torch_, nbytes, device)

    def none(torch_, nbytes, device):
        if nbytes > 0:
            raise torch.OutOfMemoryError("none left")
        return None

    want = oracle.assign(Xh, Ch)
    monkeypatch.setattr(L, "_workspace", none)
    np.testing.assert_array_equal(L.assign(X, C)[0].cpu().numpy(), want)
    np.testing.assert_array_equal(L.batch_assign(X, [0, 7, 5000], C)[0].cpu().numpy(), want)
    np.testing.assert_array_equal(h.assign(X)[0].cpu().numpy(), want)
    with pytest.raises(torch.OutOfMemoryError):
        L.assign(X, C, precision="fp16")
    monkeypatch.setattr(L, "_workspace", short)
    assert L.lloyd(X, C.clone(), 3, -1.0)["n_iter"] == 3
    assert L.lloyd_host([Xh], C.clone(), 3, -1.0)["n_iter"] == 3
