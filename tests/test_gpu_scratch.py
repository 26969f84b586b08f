"""Calls that use scratch memory only to be faster still run where the device has no room for it."""
import gc

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _fill(leave):
    """A block of device memory that leaves about `leave` bytes."""
    gc.collect()
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(max(free - leave, 0), dtype=torch.uint8, device=DEV)


def test_ranked_chi2_without_room_for_its_bins(ctx):
    """5500 locations: 3.0e7 pairs, whose bins take 0.36 GB."""
    import microsn_gb300 as mlc
    n = 5500
    rng = np.random.default_rng(1)
    A, B = (torch.as_tensor(np.exp(rng.normal(0, 0.5, (n, 3))), device=DEV) for _ in range(2))
    dA, dB = torch.diff(A, dim=1).contiguous(), torch.diff(B, dim=1).contiguous()
    v = mlc.Chi2Vars(2, np.array([0, 1], np.int32), np.array([1, 0], np.int32), np.array([0.3, 0.6]), np.array([0.2, 0.9]),
                     np.array([0.7, 1.2]), np.array([0.1, 0.2]), 0.0)
    rank, _, _ = mlc.setup_integral(ctx, A, B, mlc.bin_edges(10, 1e-2, 1e2))
    want = mlc.calculate_chi2(ctx, v, A, dA, B, dB, rank)
    spare = torch.empty_like(want)
    c = mlc.Context(0)  # without workspaces yet
    try:
        mlc.calculate_chi2(c, v, A[:50].contiguous(), dA[:50].contiguous(), B[:50].contiguous(), dB[:50].contiguous())
        del spare  # (torch keeps the block for the result)
        block = _fill(150 << 20)
        got = mlc.calculate_chi2(c, v, A, dA, B, dB, rank)
        c.synchronize()
        assert torch.equal(got, want)
        del block
    finally:
        block = None
        c.close()
        torch.cuda.empty_cache()


def test_flux_ratio_without_room_for_its_layout(ctx):
    """3300 locations of 9000 values: the large form's arrays take 0.24 GB."""
    import microsn_gb300 as mlc
    N, F, T = 3300, 9, 1000
    rng = np.random.default_rng(2)
    fo = rng.uniform(0.8, 1.2, (F, T)).astype(np.float32)
    dfo = rng.uniform(5.0, 20.0, (F, T)).astype(np.float32)
    mu = [torch.rand((N, F, T), device=DEV) + 0.5 for _ in range(2)]
    want, chi2 = mlc.flux_ratio_chi2(ctx, fo, dfo, *mu, want_chi2=True)
    c = mlc.Context(0)
    try:
        mlc.flux_ratio_chi2(c, fo[:, :2].copy(), dfo[:, :2].copy(), *[m[:80, :, :2].contiguous() for m in mu])
        block = _fill(100 << 20)
        got, got2 = mlc.flux_ratio_chi2(c, fo, dfo, *mu, want_chi2=False), None
        # FP32 terms of either form: 2^-24 of some 9000 terms each
        assert abs(got - want) <= 1e-3 * want
        del block
    finally:
        block = None
        c.close()
        torch.cuda.empty_cache()
