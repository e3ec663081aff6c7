"""One tile shape per Lloyd run: a shape that becomes the current one in the
middle of a run (here from the progress callback, as km_tune_tiles on another
thread would store it) changes neither the tables that the center bounds are
laid out for nor the results.  The later shapes have more center tiles than a
unit's mask has bits, or units of another size.  A shape that is current before
the run is the run's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _data(n, d, k):
    rng = np.random.default_rng(n + k)
    X = np.repeat(4.0 * rng.normal(size=(n // 120 + 1, d)), 120, axis=0)[:n] + 0.3 * rng.normal(size=(n, d))
    X = X.astype(np.float32)
    return X, X[rng.choice(n, size=k, replace=False)].copy()


@pytest.mark.parametrize("n,d,k,later", [
    (9000, 64, 2200, dict(bn=64, pair=0, stages=4, list_len=8)),    # 35 tiles
    (9000, 64, 2200, dict(bn=128, pair=0, stages=4, list_len=16)),
    (10001, 130, 600, dict(bn=256, pair=0, stages=2, list_len=8)),  # units of 128 frames instead of 256
    (5000, 33, 4500, dict(bn=128, pair=0, stages=3, list_len=8))])  # 36 tiles
def test_shape_stored_in_mid_run(oracle, monkeypatch, n, d, k, later):
    import torch
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_TC_BOUNDS", "1")
    X, C0 = _data(n, d, k)
    C = torch.from_numpy(C0).cuda()
    entering = [C0]

    def progress():
        entering.append(C.cpu().numpy())
        L.force_tile_plan(later)

    try:
        r = L.lloyd(torch.from_numpy(X).cuda(), C, 4, -1.0, precision="fp16", callback=progress)
    finally:
        L.force_tile_plan(None)
    np.testing.assert_array_equal(r["labels"].cpu().numpy(), oracle.assign(X, entering[3]))
    assert len(entering) == 5


@pytest.mark.parametrize("n,d,k,plan", [
    (9000, 64, 1500, dict(bn=64, pair=0, stages=4, list_len=8)),    # 24 tiles
    (9000, 64, 2200, dict(bn=64, pair=0, stages=4, list_len=8)),    # 35: no bounds
    (10001, 130, 600, dict(bn=256, pair=1, stages=3, list_len=8)),
    (10001, 130, 600, dict(bn=128, pair=0, stages=2, list_len=16))])
def test_shape_of_the_run(oracle, monkeypatch, n, d, k, plan):
    import torch
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_TC_BOUNDS", "1")
    X, C0 = _data(n, d, k)
    L.force_tile_plan(plan)
    try:
        C, entering = torch.from_numpy(C0).cuda(), [C0]
        r = L.lloyd(torch.from_numpy(X).cuda(), C, 3, -1.0, precision="fp16",
                    callback=lambda: entering.append(C.cpu().numpy()))
        np.testing.assert_array_equal(r["labels"].cpu().numpy(), oracle.assign(X, entering[2]))
    finally:
        L.force_tile_plan(None)
