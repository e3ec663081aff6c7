"""Room that the tensor-core passes reserve beside their lists: the second
pass's copies and bit table where that pass can run, within a fixed limit, and
the center bounds where a run of that size can keep them; and labels where the
limit leaves most of the overflowing frames to the full re-check."""
import numpy as np
import pytest

FP16, BF16, FP8 = 1, 3, 4
MB = 1 << 20


def _lists(n, d, k, esize=2):
    """Frame copy, candidate lists and center operands of a 16-bit pass."""
    kp = (d + 2 + 63) // 64 * 64
    return n * (kp * 2 + 16 + 172) + (k + 256) * (kp * 2 + 16)


@pytest.mark.parametrize("n,d,k", [(10_000_000, 64, 100_000), (1_000_000, 64, 1 << 20), (4_000_000, 32, 20_000)])
def test_second_pass_is_bounded(kmlib, n, d, k):
    kp = (d + 2 + 63) // 64 * 64
    most = 256 * MB + (n // 16 + 256) * (kp * 2 + 24) + 12 * n + 8 * MB  # bits, copies, lists of the rest
    for prec in (FP16, BF16):
        assert kmlib.km_assign_workspace_size(n, d, k, prec) <= _lists(n, d, k) + most


def test_second_pass_only_where_it_runs(kmlib):
    for n, d, k, prec in ((1_000_000, 528, 5000, FP8), (50_000, 128, 500, FP16), (1_000_000, 32, 1000, BF16)):
        assert kmlib.km_assign_workspace_size(n, d, k, prec) <= _lists(n, d, k) + 8 * MB


def test_bounds_only_where_they_can_be_kept(kmlib):
    def lloyd(n, d, k, prec):
        return kmlib.km_lloyd_workspace_size(n, d, k, prec) - kmlib.km_assign_workspace_size(n, d, k, prec) \
            - kmlib.km_update_workspace_size(n, d, k) - 12 * n - 4 * k * d
    assert lloyd(2_000_000, 528, 2000, FP16) >= 4 * 2_000_000
    # more tiles than a mask has bits, FP8, too little work
    for n, d, k, prec in ((1_000_000, 64, 100_000, FP16), (2_000_000, 528, 2000, FP8), (1_000_000, 64, 300, FP16)):
        assert lloyd(n, d, k, prec) <= MB


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["fp16", "bf16"])
def test_labels_at_the_limit_of_the_bit_table(prec):
    import torch
    from pyemma_gb300 import _lib as L
    g = torch.Generator(device="cuda").manual_seed(3)
    n, d, k = 300_000, 32, 1 << 17  # room for 16,128 of the 18,944 frames of a sixteenth
    means = 5.0 * torch.randn((2000, d), generator=g, device="cuda")
    C = means[torch.randint(0, 2000, (k,), generator=g, device="cuda")]
    C = (C + 1e-4 * torch.randn((k, d), generator=g, device="cuda")).contiguous()
    C[100:140] = C[7]
    X = means[torch.randint(0, 2000, (n,), generator=g, device="cuda")]
    X = (X + 0.2 * torch.randn((n, d), generator=g, device="cuda")).contiguous()
    want = L.assign(X, C, precision="fp32")[0]
    got, stats = L.assign(X, C, precision=prec)
    assert stats["n_full"] > 18_944
    assert torch.equal(got, want)
