"""Labels of Lloyd runs to the last one: a progress callback keeps the centers
that enter each iteration, and the labels of the last are the oracle's for
them, ties included.  Tensor-core passes with center bounds (both tile forms,
crowded lists with the second pass), coordinate frames with stored and with
computed features, runs in one cooperative launch, and single frames."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _last_labels(run, C0, iters):
    """run(C, progress) -> labels; (labels, centers entering the last iteration)."""
    import torch
    C, entering = torch.from_numpy(C0).cuda(), [C0]
    labels = run(C, lambda: entering.append(C.cpu().numpy()))
    assert len(entering) == iters + 1
    return labels.cpu().numpy(), entering[iters - 1]


def _dwelling(n, d, states, rng):
    means = 4.0 * rng.normal(size=(states, d))
    which = np.repeat(rng.integers(0, states, size=n // 150 + 1), 150)[:n]
    return (means[which] + 0.3 * rng.normal(size=(n, d))).astype(np.float32)


@pytest.mark.parametrize("pair", ["0", "1"])
@pytest.mark.parametrize("wide", ["0", "1"])
@pytest.mark.parametrize("prec,n,d,k,iters", [
    ("fp16", 20000, 64, 600, 5), ("fp16", 10001, 130, 1025, 4), ("bf16", 9999, 96, 520, 4), ("fp16", 300, 40, 290, 4),
    ("fp16", 12000, 700, 300, 4), ("fp16", 4000, 32, 4000, 4)])
def test_bounded_passes(oracle, monkeypatch, pair, wide, prec, n, d, k, iters):
    import torch
    from pyemma_gb300 import _lib as L
    monkeypatch.setenv("KM_TC_BOUNDS", "1")
    monkeypatch.setenv("KM_TC_PAIR", pair)
    monkeypatch.setenv("KM_TC_WIDE", wide)
    rng = np.random.default_rng(n + k)
    X = _dwelling(n, d, 40, rng)
    X[n // 3:n // 3 + 100] = X[5]  # ties
    C0 = X[rng.choice(n, size=k, replace=False)].copy()
    C0[1] = C0[0]
    C0[k // 2:k // 2 + 20] = C0[3] + 1e-5 * rng.normal(size=(20, d)).astype(np.float32)
    Xd = torch.from_numpy(X).cuda()
    got, C = _last_labels(lambda C, p: L.lloyd(Xd, C, iters, -1.0, precision=prec, callback=p)["labels"], C0, iters)
    np.testing.assert_array_equal(got, oracle.assign(X, C))


@pytest.mark.parametrize("stored", [True, False])
@pytest.mark.parametrize("prec", ["fp32", "fp16", "auto"])
@pytest.mark.parametrize("n,n_atoms,k", [(1, 3, 1), (700, 5, 7), (3001, 33, 50), (5000, 40, 300)])
def test_pair_rows(oracle, monkeypatch, stored, prec, n, n_atoms, k):
    import torch
    from pyemma_gb300 import _lib as L
    iters = 3
    rng = np.random.default_rng(n)
    xyz = torch.from_numpy(rng.normal(size=(n, n_atoms, 3)).astype(np.float32)).cuda()
    pairs = torch.tensor([(a, b) for a in range(n_atoms) for b in range(a + 1, n_atoms)], dtype=torch.int32).cuda()
    X = L.pair_distances(xyz, pairs).cpu().numpy()
    C0 = X[rng.integers(0, n, size=k)] + np.float32(0.01) * rng.normal(size=(k, X.shape[1])).astype(np.float32)
    if not stored:
        lib = L.load()
        room = L._workspace
        most = lib.km_lloyd_workspace_size(n, len(pairs), k, L.precision_code(prec))

        def short(torch_, nbytes, device):
            if nbytes > most:
                raise torch.OutOfMemoryError("none left")
            return room(torch_, nbytes, device)

        monkeypatch.setattr(L, "_workspace", short)
    got, C = _last_labels(lambda C, p: L.lloyd_pairs(xyz, pairs, C, iters, -1e9, precision=prec, callback=p)["labels"],
                          C0, iters)
    np.testing.assert_array_equal(got, oracle.assign(X, C))


@pytest.mark.parametrize("n,d,k", [(1, 1, 1), (1, 4, 3), (511, 2, 7), (20000, 5, 33), (30000, 16, 200), (200000, 2, 900)])
def test_cooperative_runs(oracle, n, d, k):
    import torch
    from pyemma_gb300 import _lib as L
    rng = np.random.default_rng(n + d + k)
    X = (rng.normal(size=(n, d)) + 4.0 * rng.integers(0, 4, size=(n, 1))).astype(np.float32)
    C0 = X[rng.integers(0, n, size=k)] + np.float32(0.01) * rng.normal(size=(k, d)).astype(np.float32)
    Xd = torch.from_numpy(X).cuda()
    got, C = _last_labels(lambda C, p: L.lloyd(Xd, C, 4, -1e9, precision="fp32", callback=p)["labels"], C0, 4)
    np.testing.assert_array_equal(got, oracle.assign(X, C))
