"""The z rank above the size from which the keys' range is looked at before they are sorted by it:
zeros, infinities and NaN of both signs, quotients of counts, all one value."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _curves(kind, n):
    rng = np.random.default_rng(n)
    A, B = (np.exp(rng.normal(0, 1, (n, 1))) for _ in range(2))
    if kind in ("zeros", "all"):
        A[::17] = 0.0
    if kind in ("infinities", "all"):
        B[5::23] = 0.0
    if kind in ("nan", "all"):
        A[7::29] = np.nan
    if kind == "all":
        A[3::19] *= -1
        A[2::19] = -0.0
        B[11::31] = -np.inf
    if kind == "counts":  # equal fractions that differ in the last bits
        A, B = (rng.poisson(300.0, (n, 1)) / 311.0 for _ in range(2))
    if kind == "one value":
        A, B = np.ones((n, 1)), np.full((n, 1), 3.0)
    return [torch.as_tensor(np.repeat(x, 3, 1), device=DEV).contiguous() for x in (A, B)]


@pytest.mark.parametrize("kind", ["zeros", "infinities", "nan", "all", "counts", "one value"])
@pytest.mark.parametrize("n", [1100, 4097])  # below and above 2^24 pairs
def test_rank_is_the_stable_order(ctx, kind, n):
    import microsn_gb300 as mlc
    A, B = _curves(kind, n)
    edges = mlc.bin_edges(60, 1e-3, 1e3)
    rank, lower, nper = mlc.setup_integral(ctx, A, B, edges)
    u = (A[:, 0][:, None] / B[:, 0][None, :]).reshape(-1).view(torch.int64)
    u[u == torch.iinfo(torch.int64).min] = 0  # -0.0 ranks as +0.0
    key = u ^ ((u >> 63) & torch.iinfo(torch.int64).max)  # the order of the bits with the sign folded in
    _, order = torch.sort(key, stable=True)
    want = torch.empty_like(order)
    want[order] = torch.arange(order.numel(), device=DEV)
    assert torch.equal(rank.to(torch.int64) & 0xFFFFFFFF, want)


# runs of equal top bits at the limits of their sorts: 2048 keys in shared memory, tiles of 8192
# through the second buffers up to 2^18, longer ones by themselves (1024 pairs per value of A)
@pytest.mark.parametrize("sizes", [[2, 3, 2, 5, 8, 9, 16, 17, 24], [255, 256, 257], [1, 2, 257, 300], [1000]])
def test_long_runs_at_their_limits(ctx, sizes):
    import microsn_gb300 as mlc
    n = 1024
    rng = np.random.default_rng(len(sizes))
    v = np.concatenate([np.full(m, 1.0 + 0.1 * i) for i, m in enumerate(sizes)])
    v = np.concatenate([v, 5.0 + np.linspace(0, 1, n - v.size)])
    v = rng.permutation(v) * (1 + 2.0 ** -45 * rng.integers(0, 5, n)) * (1 + 2.0 ** -50 * rng.integers(0, 300, n))
    A = torch.as_tensor(np.repeat(v[:, None], 3, 1), device=DEV).contiguous()
    B = torch.ones((n, 3), dtype=torch.float64, device=DEV)
    rank, _, _ = mlc.setup_integral(ctx, A, B, mlc.bin_edges(10, 1e-3, 1e3))
    _, order = torch.sort((A[:, 0][:, None] / B[:, 0][None, :]).reshape(-1), stable=True)
    want = torch.empty_like(order)
    want[order] = torch.arange(order.numel(), device=DEV)
    assert torch.equal(rank.to(torch.int64) & 0xFFFFFFFF, want)


# quotients of counts: long runs wherever fractions of different counts are equal
@pytest.mark.parametrize("n", [1100, 1500, 2200, 3000])
def test_counts_rank_no_slower_than_by_all_bits(ctx, n):
    import microsn_gb300 as mlc
    A, B = _curves("counts", n)
    edges = mlc.bin_edges(60, 1e-3, 1e3)
    z = (A[:, 0][:, None] / B[:, 0][None, :]).reshape(-1).contiguous()

    def sorting(call):
        times = []
        for _ in range(6):
            ctx.kernel_times()
            call()
            times.append(sum(ms for k, (ms, _) in ctx.kernel_times().items() if k.startswith("sort_")))
        return np.median(times[1:])

    def by_all_bits():
        mlc.sort_f64_u32(ctx, z.clone(), torch.arange(n * n, dtype=torch.int32, device=DEV))

    ctx.set_timing(True)
    try:
        assert sorting(lambda: mlc.setup_integral(ctx, A, B, edges)) <= sorting(by_all_bits)
    finally:
        ctx.set_timing(False)
