"""The calls that programs built on this package spend their time in.

Every case names a ``kind`` (which call) and its sizes.  The sizes are those
of the workloads of ``bench.py`` and the tests: low-dimensional projections
(d up to 24, as after a TICA), 528 C-alpha pair distances of a 33-bead chain,
the wide end of the precision sweep (d = 1024), chains of 58 atoms for the
minRMSD metric.

Frames lie on the GPU in all kinds but ``assign_host`` and ``fit_small``,
which take numpy arrays as PyEMMA's users hold them.
"""
import math

import numpy as np
import torch

from pyemma_gb300 import _lib, coordinates

ITERATIONS = 10  # cluster_kmeans' default max_iter
MAX_CENTERS = 2_000  # of the regular space clusterings


def listed():
    return [
        # One short request against a resident center set: launches and latency.
        dict(name="assign_tiny", kind="assign", data="low", n=1_000, d=2, k=100, precision="auto"),
        # Discretizing a TICA projection: 20 trajectories of uneven length.
        dict(name="assign_low", kind="assign", data="low", n=2_000_003, d=4, k=500, precision="auto"),
        # Discretizing C-alpha distances with converged centers (the headline's shape).
        dict(name="assign_wide", kind="assign", data="chain", n=2_000_000, d=528, k=2_000, precision="auto"),
        # Odd sizes at the wide end: rows that are no multiple of 16 bytes.
        dict(name="assign_ragged", kind="assign", data="mixture", n=250_007, d=1_023, k=777, precision="auto"),
        # assign_to_centers on ordinary numpy arrays, dtrajs back in host memory.
        dict(name="assign_host", kind="assign_host", n=400_000, d=528, k=500, n_traj=8),
        # The whole cluster_kmeans call at tutorial size: kmeans++ and Lloyd to convergence.
        dict(name="fit_small", kind="fit_small", n=100_000, d=2, k=50, max_iter=100),
        # Lloyd iterations on low-dimensional trajectories, from given centers.
        dict(name="fit_low", kind="fit", data="low", n=4_280_267, d=10, k=1_000),
        # Lloyd iterations on C-alpha distances (the headline), from given centers.
        dict(name="fit_wide", kind="fit", data="chain", n=2_000_000, d=528, k=2_000),
        # The same model from coordinates: features computed where they are read.
        dict(name="fit_pairs", kind="fit_pairs", n=500_000, d=528, k=1_000),
        # kmeans++ on C-alpha distances.
        dict(name="kmpp_wide", kind="kmpp", n=500_000, d=528, k=300),
        # Assignment by RMSD after superposition, with the distances.
        dict(name="minrmsd", kind="minrmsd", n=1_000_000, d=174, k=100),
        # Regular space clustering of a TICA projection.
        dict(name="regspace", kind="regspace", n=1_000_000, d=3, dmin=1.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["assign_low", "assign_low", "assign_chain", "assign_mixture", "assign_host", "fit_small",
                       "fit_low", "fit_low", "fit_mixture", "fit_chain", "fit_pairs", "kmpp", "minrmsd", "regspace"])
    if kind == "assign_low":
        return dict(kind="assign", data="low", n=_log(rng, 1_000, 4_000_000), d=rng.randint(1, 24),
                    k=_log(rng, 50, 2_000), precision=rng.choice(["auto", "auto", "auto", "fp16", "fp32"]))
    if kind == "assign_chain":
        return dict(kind="assign", data="chain", n=_log(rng, 2_000, 2_000_000), d=528, k=_log(rng, 100, 2_000),
                    precision=rng.choice(["auto", "auto", "fp16", "bf16"]))
    if kind == "assign_mixture":
        return dict(kind="assign", data="mixture", n=_log(rng, 5_000, 250_000), d=_log(rng, 25, 1_024),
                    k=_log(rng, 50, 2_000), precision=rng.choice(["auto", "auto", "fp16", "bf16"]))
    if kind == "assign_host":
        return dict(kind="assign_host", n=_log(rng, 5_000, 400_000), d=rng.choice([3, 10, 33, 528]),
                    k=_log(rng, 50, 1_000), n_traj=rng.randint(1, 12))
    if kind == "fit_small":
        return dict(kind="fit_small", n=_log(rng, 2_000, 200_000), d=rng.randint(1, 6), k=_log(rng, 5, 120),
                    max_iter=rng.choice([10, 50, 100]))
    if kind == "fit_low":
        return dict(kind="fit", data="low", n=_log(rng, 20_000, 4_280_267), d=rng.randint(2, 24),
                    k=_log(rng, 50, 1_000))
    if kind == "fit_mixture":
        return dict(kind="fit", data="mixture", n=_log(rng, 20_000, 250_000), d=_log(rng, 25, 1_024),
                    k=_log(rng, 50, 1_000))
    if kind == "fit_chain":
        return dict(kind="fit", data="chain", n=_log(rng, 50_000, 2_000_000), d=528, k=_log(rng, 200, 2_000))
    if kind == "fit_pairs":
        return dict(kind="fit_pairs", n=_log(rng, 20_000, 500_000), d=528, k=_log(rng, 100, 1_000))
    if kind == "kmpp":
        return dict(kind="kmpp", n=_log(rng, 20_000, 500_000), d=rng.choice([4, 10, 67, 528]), k=_log(rng, 20, 300))
    if kind == "minrmsd":
        return dict(kind="minrmsd", n=_log(rng, 5_000, 1_000_000), d=3 * rng.randint(5, 58), k=_log(rng, 10, 100))
    return dict(kind="regspace", n=_log(rng, 20_000, 1_000_000), d=3, dmin=round(rng.uniform(1.0, 2.5), 2))


# ---- inputs -----------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1_000_003 + seed)


def _dwell_states(n, n_states, mean_dwell, rng):
    """A state per frame, changing after geometric waiting times."""
    waits = rng.geometric(1.0 / mean_dwell, size=2 * (n // mean_dwell) + 4)
    starts = np.cumsum(np.concatenate([[0], waits]))
    states = rng.integers(0, n_states, size=len(starts))
    return states[np.searchsorted(starts, np.arange(n), side="right") - 1]


def _low_frames(n, d, seed):
    """AR(1) fluctuations (0.995, 0.1) about 8 metastable means U[-3, 3]^d with jumps every ~5,000 frames."""
    rng = np.random.default_rng(seed)
    a, block = 0.995, 1_000
    means = torch.from_numpy(rng.uniform(-3.0, 3.0, size=(8, d))).cuda()
    states = torch.from_numpy(_dwell_states(n, 8, 5_000, rng)).cuda()
    nb = -(-n // block)
    eps = 0.1 * torch.randn((nb, block, d), generator=_gen(seed), device="cuda", dtype=torch.float64)
    # y_t = a y_{t-1} + eps_t: blocks by scaled cumulative sums, then the carry from block to block
    power = a ** torch.arange(block, device="cuda", dtype=torch.float64)[:, None]
    y = torch.cumsum(eps / power, dim=1) * power
    last = y[:, -1].cpu().numpy()
    carry = np.zeros((nb, d))
    for b in range(1, nb):
        carry[b] = last[b - 1] + a ** block * carry[b - 1]
    y += torch.from_numpy(carry).cuda()[:, None, :] * (power * a)
    return (means[states] + y.reshape(nb * block, d)[:n]).float().contiguous()


def _chain_coordinates(n, n_beads, bond, jitter, n_conf, seed):
    """Jittered copies of random-walk chains, dwelling ~2,000 frames in each conformation."""
    rng = np.random.default_rng(seed)
    steps = rng.standard_normal((n_conf, n_beads - 1, 3))
    steps *= bond / np.linalg.norm(steps, axis=2, keepdims=True)
    base = np.concatenate([np.zeros((n_conf, 1, 3)), np.cumsum(steps, axis=1)], axis=1)
    conf = torch.from_numpy(_dwell_states(n, n_conf, 2_000, rng)).cuda()
    xyz = jitter * torch.randn((n, n_beads, 3), generator=_gen(seed), device="cuda")
    xyz += torch.from_numpy(base).float().cuda()[conf]
    return xyz


def _all_pairs(n_beads):
    i, j = np.triu_indices(n_beads, k=1)
    return np.stack([i, j], axis=1).astype(np.int32)


def _chain_distances(n, seed):
    """All 528 pair distances of a 33-bead chain (0.38 nm bonds, 0.05 nm jitter)."""
    xyz = _chain_coordinates(n, 33, 0.38, 0.05, 64, seed)
    pairs = torch.from_numpy(_all_pairs(33)).long().cuda()
    out = torch.empty((n, len(pairs)), device="cuda")
    for a in range(0, n, 1 << 17):
        part = xyz[a:a + (1 << 17)]
        out[a:a + (1 << 17)] = (part[:, pairs[:, 1]] - part[:, pairs[:, 0]]).square().sum(-1).sqrt()
    return out


def _mixture(n, d, k, seed):
    """4k Gaussian clusters of sigma 0.3 with means U[-5, 5]^d."""
    g = _gen(seed)
    means = 10.0 * torch.rand((4 * k, d), generator=g, device="cuda") - 5.0
    which = torch.randint(0, 4 * k, (n,), generator=g, device="cuda")
    X = 0.3 * torch.randn((n, d), generator=g, device="cuda")
    X += means[which]
    return X


def _frames(case, seed):
    if case["data"] == "low":
        return _low_frames(case["n"], case["d"], seed)
    if case["data"] == "chain":
        return _chain_distances(case["n"], seed)
    return _mixture(case["n"], case["d"], case["k"], seed)


def _mean_centers(X, k, seed):
    """Centers as an estimate leaves them: means of near frames (here runs of 16 consecutive ones)."""
    rng = np.random.default_rng(seed + 17)
    first = torch.from_numpy(rng.integers(0, max(1, len(X) - 16), size=k)).cuda()
    C = torch.zeros((k, X.shape[1]), device="cuda")
    for t in range(16):
        C += X[torch.clamp(first + t, max=len(X) - 1)]
    return (C / 16.0).contiguous()


def _first_centers(X, k, seed):
    rng = np.random.default_rng(seed + 29)
    rows = np.sort(rng.choice(len(X), size=k, replace=False))
    return X[torch.from_numpy(rows).cuda()].contiguous()


def _rotations(n, g):
    q = torch.randn((n, 4), generator=g, device="cuda")
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    rows = [1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
            2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
            2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)]
    return torch.stack(rows, dim=1).view(n, 3, 3)


def _tumbling_chains(n, n_atoms, n_chains, seed):
    """Noisy copies of random-walk chains, randomly rotated and translated."""
    g = _gen(seed)
    steps = torch.randn((n_chains, n_atoms, 3), generator=g, device="cuda")
    base = torch.cumsum(3.8 * steps / steps.norm(dim=2, keepdim=True), dim=1)
    which = torch.randint(0, n_chains, (n,), generator=g, device="cuda")
    pos = 0.8 * torch.randn((n, n_atoms, 3), generator=g, device="cuda")
    pos += base[which]
    X = torch.matmul(pos, _rotations(n, g).transpose(1, 2))
    X += 10.0 * torch.randn((n, 1, 3), generator=g, device="cuda")
    return X.reshape(n, 3 * n_atoms).contiguous()


def prepare(case, seed):
    kind, n, d, k = case["kind"], case["n"], case["d"], case.get("k")
    if kind == "assign":
        X = _frames(case, seed)
        # a program that assigns many trajectories keeps its centers resident
        return dict(case=case, X=X, centers=_lib.Centers(_mean_centers(X, k, seed), precision=case["precision"]))
    if kind == "assign_host":
        X = _chain_distances(n, seed) if d == 528 else _low_frames(n, d, seed)
        C = _mean_centers(X, k, seed).cpu().numpy()
        cuts = np.sort(np.random.default_rng(n).integers(0, n + 1, size=case["n_traj"] - 1))
        return dict(case=case, trajs=[np.ascontiguousarray(t) for t in np.split(X.cpu().numpy(), cuts) if len(t)], C=C)
    if kind == "fit_small":
        g = _gen(seed)
        means = 10.0 * torch.rand((10, d), generator=g, device="cuda") - 5.0
        X = means[torch.randint(0, 10, (n,), generator=g, device="cuda")]
        return dict(case=case, X=(X + 0.5 * torch.randn((n, d), generator=g, device="cuda")).cpu().numpy())
    if kind == "fit":
        X = _frames(case, seed)
        return dict(case=case, X=X, C0=_first_centers(X, k, seed).cpu().numpy())
    if kind == "fit_pairs":
        from pyemma_gb300.featurize import pair_distance_frames
        frames = pair_distance_frames(_chain_coordinates(n, 33, 0.38, 0.05, 64, seed), pairs=_all_pairs(33))
        rows = np.sort(np.random.default_rng(seed + 29).choice(n, size=k, replace=False))
        xyz = frames.xyz[torch.from_numpy(rows).cuda()]
        pairs = torch.from_numpy(_all_pairs(33)).long().cuda()
        C0 = (xyz[:, pairs[:, 1]] - xyz[:, pairs[:, 0]]).square().sum(-1).sqrt()
        return dict(case=case, frames=frames, C0=C0.cpu().numpy())
    if kind == "kmpp":
        X = _chain_distances(n, seed) if d == 528 else _low_frames(n, d, seed)
        return dict(case=case, X=X, seed=42)
    if kind == "minrmsd":
        X = _tumbling_chains(n, d // 3, k, seed)
        return dict(case=case, X=X, C=_first_centers(X, k, seed))
    return dict(case=case, X=_low_frames(n, d, seed))


# ---- one pass ---------------------------------------------------------------
def _model(est):
    return dict(centers=est.clustercenters, inertias=est.inertias)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "assign":
        return state["centers"].assign(state["X"])[0]
    if kind == "assign_host":
        return coordinates.assign_to_centers(state["trajs"], centers=state["C"])
    if kind == "fit_small":
        est = coordinates.cluster_kmeans(state["X"], k=case["k"], max_iter=case["max_iter"], fixed_seed=42)
        return dict(centers=est.clustercenters, inertia=float(est.inertias[-1]))
    if kind == "fit":
        # tolerance 0: all iterations run, as in the benchmark
        return _model(coordinates.cluster_kmeans(state["X"], k=case["k"], max_iter=ITERATIONS, tolerance=0.0,
                                                 clustercenters=state["C0"]))
    if kind == "fit_pairs":
        return _model(coordinates.cluster_kmeans(state["frames"], k=case["k"], max_iter=ITERATIONS, tolerance=0.0,
                                                 clustercenters=state["C0"]))
    if kind == "kmpp":
        C0, idx = _lib.kmpp(state["X"], case["k"], state["seed"])
        return dict(centers=C0, frames=idx)
    if kind == "minrmsd":
        labels, rmsd = _lib.assign_minrmsd(state["X"], state["C"], return_rmsd=True)
        return dict(labels=labels, rmsd=rmsd)
    est = coordinates.cluster_regspace(state["X"], dmin=case["dmin"], max_centers=MAX_CENTERS)
    centers = np.zeros((MAX_CENTERS, case["d"]), dtype=np.float32)
    centers[:len(est.clustercenters)] = est.clustercenters  # their number depends on the frames
    return dict(centers=centers, dtraj=est.dtrajs[0])


def work(case):
    kind, n, d, k = case["kind"], case["n"], case["d"], case.get("k") or 1
    frames = 4.0 * n * d
    if kind in ("assign", "assign_host"):
        return dict(bytes=frames + 4.0 * k * d + 4.0 * n, flops=2.0 * n * k * d)
    if kind == "fit":
        # the frames are read again by every iteration unless the 129 MB L2 holds them
        reads = ITERATIONS if frames > 129e6 else 1
        return dict(bytes=reads * frames + 8.0 * k * d, flops=2.0 * n * k * d * ITERATIONS)
    if kind == "fit_pairs":
        xyz = 12.0 * n * 33
        return dict(bytes=(ITERATIONS if xyz > 129e6 else 1) * xyz + 8.0 * k * d, flops=2.0 * n * k * d * ITERATIONS)
    if kind == "fit_small":
        return dict(bytes=frames + 4.0 * k * d, flops=2.0 * n * k * d)
    if kind == "kmpp":
        # every center is a row; a row of a frame that no center can reach is read once
        return dict(bytes=frames + 4.0 * k * d + 8.0 * k, flops=3.0 * n * d)
    if kind == "minrmsd":
        return dict(bytes=frames + 4.0 * k * d + 8.0 * n, flops=6.0 * n * k * d)
    return dict(bytes=frames + 4.0 * n, flops=3.0 * n * d)


# ---- the same in 64 bits ----------------------------------------------------
def _lloyd64(X, C0, iterations):
    C = torch.from_numpy(C0).cuda().double()
    k = len(C)
    inertias = []
    rows = max(1, int(5e7) // k)
    for _ in range(iterations):
        sums = torch.zeros_like(C)
        counts = torch.zeros(k, device="cuda", dtype=torch.float64)
        half = 0.5 * C.square().sum(1)
        labels = []
        for a in range(0, len(X), rows):
            part = X[a:a + rows].double()
            lab = (part @ C.T - half).argmax(1)
            sums.index_add_(0, lab, part - C[lab])
            counts += torch.bincount(lab, minlength=k)
            labels.append(lab)
        C = C + sums / counts.clamp(min=1)[:, None]
        inertia = 0.0
        for a, lab in zip(range(0, len(X), rows), labels):
            inertia += float((X[a:a + rows].double() - C[lab]).square().sum())
        inertias.append(inertia)
    return dict(centers=C.cpu().numpy(), inertias=np.array(inertias))


def _rmsd64(X, C):
    """sqrt of the smallest mean square deviation after optimal superposition."""
    n, k, m = len(X), len(C), X.shape[1] // 3
    out = torch.empty(n, device="cuda", dtype=torch.float64)
    B = C.double().view(k, m, 3)
    B = B - B.mean(1, keepdim=True)
    gb = B.square().sum((1, 2))
    rows = max(1, int(2e6) // k)
    for a in range(0, n, rows):
        A = X[a:a + rows].double().view(-1, m, 3)
        A = A - A.mean(1, keepdim=True)
        S = torch.einsum("iap,jaq->ijpq", A, B)
        # the largest root of the characteristic polynomial of the 4x4 key matrix, by Newton's method from above
        ss = S.square().sum((2, 3))
        c2, c1 = -2.0 * ss, -8.0 * torch.linalg.det(S)
        t = S @ S.transpose(2, 3)
        c0 = 2.0 * t.square().sum((2, 3)) - ss * ss  # the product of the key matrix's eigenvalues
        lam = torch.sqrt(3.0 * ss)
        for _ in range(60):
            p = ((lam * lam + c2) * lam + c1) * lam + c0
            dp = (4.0 * lam * lam + 2.0 * c2) * lam + c1
            lam = lam - torch.where(dp != 0, p / dp, torch.zeros_like(p))
        msd = (A.square().sum((1, 2))[:, None] + gb[None, :] - 2.0 * lam) / m
        out[a:a + rows] = msd.clamp(min=0).min(1).values.sqrt()
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "minrmsd":
        state = prepare(case, seed)
        return dict(labels=None, rmsd=_rmsd64(state["X"], state["C"]))
    if kind == "fit" and case["n"] * case["k"] * case["d"] <= 1e11:
        state = prepare(case, seed)
        return _lloyd64(state["X"], state["C0"], ITERATIONS)
    return None  # labels and copies of frames, or too long in 64 bits
