"""Lloyd runs whose first iteration reports a wait that ran out: the run ends
with that status before anything reads the labels (which such a pass may leave
unwritten), with the bounds of the tensor-core pass on and off, from device and
from host frames, and the next run is as if nothing had happened.  The error is
planted on the host; no device wait is made to run out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bounds", ["0", "1"])
@pytest.mark.parametrize("host", [False, True])
def test_first_iteration_reports_a_timeout(oracle, monkeypatch, bounds, host):
    import torch
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_TC_BOUNDS", bounds)
    rng = np.random.default_rng(5)
    X = np.repeat(rng.normal(size=(60, 64)), 100, axis=0) + 0.1 * rng.normal(size=(6000, 64))
    X = X.astype(np.float32)
    C0 = X[rng.choice(6000, size=300, replace=False)].copy()

    def run(C):
        if host:
            return L.lloyd_host([X], C, 3, -1.0, precision="fp16")
        return L.lloyd(torch.from_numpy(X).cuda(), C, 3, -1.0, precision="fp16")

    assert L.load().km_debug_fake_device_error(4) == L.KM_OK
    with pytest.raises(L.KmError) as ei:
        run(torch.from_numpy(C0).cuda())
    assert ei.value.status == L.KM_ERR_TIMEOUT
    C = torch.from_numpy(C0).cuda()
    got = run(C)
    want = oracle.lloyd(X, C0, 3, -1.0)
    assert got["n_iter"] == 3
    np.testing.assert_allclose(C.cpu().numpy(), want["centers"], rtol=1e-5, atol=1e-5)
