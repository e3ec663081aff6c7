"""kmeans++ draws that a device-side wait cut short are reported: the wrappers
and the estimators raise instead of going on from NaN centers, and so do Lloyd
runs of one cooperative launch.  The error is planted on the host; no device
wait is made to run out.  Under stream capture, where nothing has run yet, the
draw is enqueued as it is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frames(n=3000, d=5):
    import torch
    return torch.from_numpy(np.random.default_rng(2).normal(size=(n, d)).astype(np.float32)).cuda()


@pytest.mark.parametrize("k", [1, 7, 64, 130])  # within a launch, at its end, over several
@pytest.mark.parametrize("prune", ["0", "1"])
def test_kmpp_reports_a_timeout(monkeypatch, k, prune):
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_KMPP_PRUNE", prune)
    X = _frames()
    want = L.kmpp(X, k, 3)[1]
    assert L.load().km_debug_fake_device_error(4) == L.KM_OK
    with pytest.raises(L.KmError) as ei:
        L.kmpp(X, k, 3)
    assert ei.value.status == L.KM_ERR_TIMEOUT
    assert bool((L.kmpp(X, k, 3)[1] == want).all())


def test_kmpp_pairs_and_estimators_report_a_timeout():
    import torch
    from pyemma_gb300 import _lib as L, coordinates, deeptime_clustering
    lib, X = L.load(), _frames()
    xyz = torch.randn((500, 6, 3), device="cuda")
    pairs = torch.tensor([[0, 1], [2, 5], [1, 4]], dtype=torch.int32, device="cuda")
    calls = (lambda: L.kmpp_pairs(xyz, pairs, 4, 1), lambda: coordinates.cluster_kmeans(X.cpu().numpy(), k=5),
             lambda: deeptime_clustering.KMeans(5).fit(X.cpu().numpy()))
    for call in calls:
        assert lib.km_debug_fake_device_error(2) == L.KM_OK
        with pytest.raises(L.KmError) as ei:
            call()
        assert ei.value.status == L.KM_ERR_TIMEOUT
        call()


def test_small_lloyd_reports_a_timeout():
    from pyemma_gb300 import _lib as L
    X = _frames()
    assert L.load().km_debug_fake_device_error(4) == L.KM_OK
    with pytest.raises(L.KmError) as ei:
        L.lloyd(X, X[:9].clone(), 5, -1.0, precision="fp32")
    assert ei.value.status == L.KM_ERR_TIMEOUT
    assert L.lloyd(X, X[:9].clone(), 5, -1.0, precision="fp32")["n_iter"] == 5


def test_kmpp_under_capture():
    import torch
    from pyemma_gb300 import _lib as L
    X = _frames()
    want = L.kmpp(X, 70, 11)[1]
    s, g = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    s.wait_stream(torch.cuda.current_stream())
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        idx = L.kmpp(X, 70, 11)[1]
    g.replay()
    torch.cuda.synchronize()
    assert bool((idx == want).all())
