"""Lloyd on coordinate frames with the features stored in the workspace (as
much as km_lloyd_pairs_workspace_size asks for) and without (the dense call's
workspace): the same run, and the caller's bytes behind the workspace stay."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp16", "auto"])
@pytest.mark.parametrize("n,n_atoms,k,iters", [(1, 3, 1, 2), (700, 5, 7, 3), (3001, 33, 50, 4), (5000, 40, 300, 2)])
def test_lloyd_pairs_with_and_without_rows(prec, n, n_atoms, k, iters):
    import torch
    from pyemma_gb300 import _lib as L
    lib = L.load()
    rng = np.random.default_rng(n)
    xyz = torch.from_numpy(rng.normal(size=(n, n_atoms, 3)).astype(np.float32)).cuda()
    pairs = torch.tensor([(a, b) for a in range(n_atoms) for b in range(a + 1, n_atoms)], dtype=torch.int32).cuda()
    d, p = len(pairs), L.precision_code(prec)
    C0 = L.pair_distances(xyz[torch.from_numpy(rng.integers(0, n, size=k)).cuda()].contiguous(), pairs)
    sizes = [lib.km_lloyd_workspace_size(n, d, k, p), lib.km_lloyd_pairs_workspace_size(n, d, k, p)]
    assert sizes[1] >= sizes[0] + 4 * n * d
    out = []
    for size in sizes:
        ws = torch.full((size + 256,), 7, dtype=torch.uint8, device="cuda")
        C, labels = C0.clone(), torch.empty(n, dtype=torch.int32, device="cuda")
        inertias, it, conv = np.zeros(iters), ctypes.c_int32(0), ctypes.c_int32(0)
        L.check(lib.km_lloyd_pairs(L._ptr(xyz), n, n_atoms, L._ptr(pairs), d, k, L._ptr(C), iters, -1.0, p,
                                   L._ptr(labels), inertias.ctypes.data_as(ctypes.c_void_p), ctypes.byref(it),
                                   ctypes.byref(conv), L._callback(None)[0], None, L._ptr(ws), size,
                                   L._stream(torch, xyz.device)))
        assert bool((ws[size:] == 7).all()) and it.value == iters
        out.append((labels.cpu().numpy(), C.cpu().numpy(), inertias))
    assert (out[0][0] != out[1][0]).sum() <= 2  # float64 sums in another order
    np.testing.assert_allclose(out[1][1], out[0][1], rtol=1e-5, atol=1e-5)
    np.testing.assert_allclose(out[1][2], out[0][2], rtol=1e-6, atol=1e-4)
