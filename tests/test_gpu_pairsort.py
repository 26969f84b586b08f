"""The sort at the edges of its one-CTA and tiled forms, the pair stage's writes in rank order
below and above the size from which they go through bins, its quotients and exponentials."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n", [2, 33, 1024, 1025, 8192, 8193, 16384, 16385, 24576, 24577, 1_000_003])
@pytest.mark.parametrize("kind", ["normal", "few", "low bits", "infinite"])
def test_sort_stable_at_tile_edges(ctx, n, kind):
    import microsn_gb300 as mlc
    rng = np.random.default_rng(n)
    k = rng.normal(0, 1, n)
    if kind == "few":
        k = np.floor(3 * k)
    elif kind == "low bits":  # one exponent, differing in the last bits only
        k = (np.float64(1.5).view(np.int64) + rng.integers(0, 300, n)).view(np.float64)
    elif kind == "infinite":
        k[::3] = np.inf; k[1::5] = -np.inf
    keys = torch.as_tensor(k, device=DEV)
    vals = torch.arange(n, dtype=torch.int32, device=DEV)
    mlc.sort_f64_u32(ctx, keys, vals)
    order = np.lexsort((np.arange(n), np.where(k == 0, np.copysign(1, k) * 1e-300, k)))
    assert np.array_equal(vals.cpu().numpy(), order.astype(np.int32))
    assert np.array_equal(keys.cpu().numpy(), k[order])


def _curves(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "integers":  # quotients with many ties and near ties
        c = rng.integers(1, 4000, (n, 3)).astype(np.float64)
    elif kind == "extreme":  # quotients that the reciprocal form leaves to the division
        c = np.exp(rng.normal(0, 1, (n, 3))) * 10.0 ** rng.integers(-150, 150, (n, 1))
    else:
        c = np.exp(rng.normal(0, 1, (n, 1)) + 0.1 * rng.normal(0, 1, (n, 3)))
    return torch.as_tensor(c, device=DEV)


# quotients in long runs of equal top bits whose keys alternate: 2, 64 and more than the 64 large
# runs that are sorted one by one, 1200 that a CTA each sorts, at the ends of the range and
# across tiles
@pytest.mark.parametrize("runs", [2, 64, 150, 1200])
def test_long_runs_out_of_order(ctx, runs):
    import microsn_gb300 as mlc
    n = 1200
    rng = np.random.default_rng(runs)
    v = np.linspace(1.0, 3.0, runs)[rng.integers(0, runs, n)]
    A = torch.as_tensor(np.repeat((v * (1 + 2.0 ** -45 * rng.integers(0, 3, n)))[:, None], 3, 1), device=DEV)
    B = torch.ones((n, 3), dtype=torch.float64, device=DEV)
    rank, _, _ = mlc.setup_integral(ctx, A.contiguous(), B, mlc.bin_edges(10, 1e-3, 1e3))
    _, order = torch.sort((A[:, 0][:, None] / B[:, 0][None, :]).reshape(-1), stable=True)
    want = torch.empty_like(order)
    want[order] = torch.arange(order.numel(), device=DEV)
    assert torch.equal(rank.to(torch.int64) & 0xFFFFFFFF, want)


# from 1024 pairs a side on the keys are sorted by the top of their range, 5600: chi2 and ranks
# written through bins (above 3e7)
@pytest.mark.parametrize("kind,n", [("integers", 300), ("extreme", 1100), ("smooth", 1500), ("integers", 1500),
                                    ("smooth", 5600)])
def test_ranked_pairs_match_torch(ctx, kind, n):
    import microsn_gb300 as mlc
    A, B = _curves(kind, n, 1), _curves(kind, n, 2)
    dA, dB = torch.diff(A, dim=1).contiguous(), torch.diff(B, dim=1).contiguous()
    edges = mlc.bin_edges(120, 1e-3, 1e3)
    rank, lower, nper = mlc.setup_integral(ctx, A, B, edges)
    z = (A[:, 0][:, None] / B[:, 0][None, :]).reshape(-1)
    zs, order = torch.sort(z, stable=True)
    want = torch.empty_like(order)
    want[order] = torch.arange(order.numel(), device=DEV)
    assert torch.equal(rank.to(torch.int64) & 0xFFFFFFFF, want)
    up = torch.searchsorted(zs, torch.as_tensor(edges, device=DEV), right=True).cpu().numpy()
    assert np.array_equal(nper, np.diff(np.concatenate([[0], up])).astype(np.uint32))
    v = mlc.Chi2Vars(3, np.array([0, 1, -1], np.int32), np.array([1, -1, 0], np.int32), np.array([0.3, 0.6, 0.0]),
                     np.array([0.2, 0.0, 0.9]), np.array([0.7, 1.2, 1.1]), np.array([0.1, 0.15, 0.3]), 0.0)
    chi2 = mlc.calculate_chi2(ctx, v, A, dA, B, dB, rank)
    ref = torch.zeros((n, n), dtype=torch.float64, device=DEV)
    cond = torch.zeros_like(ref)  # sum of what each term's rounding is relative to
    for i in range(3):
        a = A[:, v.indA[i]] + v.facA[i] * dA[:, v.indA[i]] if v.indA[i] >= 0 else torch.ones(n, dtype=torch.float64, device=DEV)
        b = B[:, v.indB[i]] + v.facB[i] * dB[:, v.indB[i]] if v.indB[i] >= 0 else torch.ones(n, dtype=torch.float64, device=DEV)
        q = a[:, None] / b[None, :]
        t = (v.d[i] - q) / v.s[i]
        ref += t * t
        cond += 2 * t.abs() * (abs(v.d[i]) + q) / v.s[i] + t * t
    err = (chi2 - ref.reshape(-1)[order]).abs()
    # a few roundings of 2^-53 of each term's operands on either side
    assert bool((err <= 8 * 2.0 ** -53 * cond.reshape(-1)[order] + 1e-300).all() | ~torch.isfinite(ref).all())
    # bin means: exponentials within a few ulp, sums of up to millions of them
    bc, be = mlc.bin_chi2(ctx, lower, nper, chi2)
    fb, fe, fn = mlc.pair_bin_fused(ctx, v, A, dA, B, dB, edges)
    assert np.array_equal(fn, nper)
    for i in np.nonzero(nper)[0]:
        part = chi2[int(lower[i]):int(lower[i]) + int(nper[i])]
        for got, g2, x in ((bc[i], fb[i], part.mean().item()), (be[i], fe[i], torch.exp(-0.5 * part).mean().item())):
            assert abs(got - x) <= 1e-13 * abs(x) + 1e-320
            assert abs(g2 - x) <= 1e-12 * abs(x) + 1e-320


def test_zero_sigma_and_data_keep_their_terms(ctx):
    """d = 0 and s = 0 take the undivided terms: the same infinities and values as (d - x)/s."""
    import microsn_gb300 as mlc
    A, B = _curves("smooth", 64, 1), _curves("smooth", 64, 2)
    dA, dB = torch.diff(A, dim=1).contiguous(), torch.diff(B, dim=1).contiguous()
    q = A[:, 0][:, None] / B[:, 1][None, :]
    for d, s in ((0.0, 0.1), (0.7, 0.0)):
        v = mlc.Chi2Vars(1, np.array([0], np.int32), np.array([0], np.int32), np.array([0.0]), np.array([1.0]),
                         np.array([d]), np.array([s]), 0.0)
        got = mlc.calculate_chi2(ctx, v, A, dA, B, dB).reshape(64, 64)
        ref = ((d - q) / s) ** 2
        assert torch.allclose(got, ref, rtol=1e-12, atol=0)
