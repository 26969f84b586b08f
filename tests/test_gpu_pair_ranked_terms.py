"""Ranked chi2 of many pairs: from six epochs on the tiles of pairs are the faster form, whose time
the scattered stores bound."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _vars(n):
    import microsn_gb300 as mlc
    r = np.random.default_rng(n)
    return mlc.Chi2Vars(n, r.integers(0, 2, n).astype(np.int32), r.integers(0, 2, n).astype(np.int32), r.random(n),
                        r.random(n), np.full(n, 1.1), np.full(n, 0.3), 0.0)


def test_more_epochs_in_rank_order(ctx):
    import microsn_gb300 as mlc
    n = 5600
    r = np.random.default_rng(1)
    A, B = (torch.as_tensor(np.exp(r.normal(0, 1, (n, 3))), device=DEV) for _ in range(2))
    dA, dB = torch.diff(A, dim=1).contiguous(), torch.diff(B, dim=1).contiguous()
    rank, _, _ = mlc.setup_integral(ctx, A, B, mlc.bin_edges(10, 1e-3, 1e3))
    at = rank.to(torch.int64) & 0xFFFFFFFF
    ms = {}
    for terms in (5, 6, 8):
        v = _vars(terms)
        want = mlc.calculate_chi2(ctx, v, A, dA, B, dB)
        assert torch.equal(mlc.calculate_chi2(ctx, v, A, dA, B, dB, rank)[at], want)
        ctx.set_timing(True)
        times = []
        for _ in range(7):
            ctx.kernel_times()
            mlc.calculate_chi2(ctx, v, A, dA, B, dB, rank)
            times.append(ctx.kernel_times()["pair_chi2_ratio"][0])
        ctx.set_timing(False)
        ms[terms] = sorted(times)[3]
    assert ms[6] <= 1.1 * ms[5] and ms[8] <= 1.15 * ms[5]


def test_few_locations_add_up_few_copies(ctx):
    """The fused bins of 10 locations: as many copies of the accumulators as CTAs, whose sum takes less
    than the pairs' kernel (1024 copies took half as long again)."""
    import microsn_gb300 as mlc
    r = np.random.default_rng(2)
    A, B = (torch.as_tensor(np.exp(r.normal(0, 1, (10, 3))), device=DEV) for _ in range(2))
    dA, dB = torch.diff(A, dim=1).contiguous(), torch.diff(B, dim=1).contiguous()
    edges = mlc.bin_edges(300, 1e-4, 300.0)
    v = _vars(3)
    mlc.pair_bin_fused(ctx, v, A, dA, B, dB, edges)
    ctx.set_timing(True)
    times = {"pair_bin_combine": [], "pair_bin_fused": []}
    for _ in range(9):
        ctx.kernel_times()
        mlc.pair_bin_fused(ctx, v, A, dA, B, dB, edges)
        t = ctx.kernel_times()
        for k in times:
            times[k].append(t[k][0])
    ctx.set_timing(False)
    assert sorted(times["pair_bin_combine"])[4] <= sorted(times["pair_bin_fused"])[4]
