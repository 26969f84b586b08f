"""The ratio chi2 where light-curve values, data or errors lie near the ends of FP64: the same
values as the undivided terms (d - a/b)/s, and the same infinities and NaN."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _vars(d, s):
    import microsn_gb300 as mlc
    return mlc.Chi2Vars(3, np.array([0, 1, -1], np.int32), np.array([1, -1, 0], np.int32), np.array([0.3, 0.6, 0.0]),
                        np.array([0.2, 0.0, 0.9]), np.array(d), np.array(s), 0.0)


def _reference(v, A, dA, B, dB):
    """chi2 of all pairs term by term, and what its rounding is relative to."""
    n = A.shape[0]
    one = torch.ones(n, dtype=torch.float64, device=DEV)
    ref = torch.zeros((n, n), dtype=torch.float64, device=DEV)
    cond = torch.zeros_like(ref)
    for i in range(v.Njp):
        a = A[:, v.indA[i]] + v.facA[i] * dA[:, v.indA[i]] if v.indA[i] >= 0 else one
        b = B[:, v.indB[i]] + v.facB[i] * dB[:, v.indB[i]] if v.indB[i] >= 0 else one
        q = a[:, None] / b[None, :]
        t = (v.d[i] - q) / v.s[i]
        ref += t * t
        cond += 2 * t.abs() * ((abs(v.d[i]) + q) / v.s[i]) + t * t
    return ref, cond


def _check(chi2, ref, cond):
    fin = torch.isfinite(ref) & torch.isfinite(cond)
    assert bool(fin.any())
    # a few roundings of 2^-53 of each term's operands on either side
    assert bool(((chi2 - ref).abs() <= 8 * 2.0 ** -53 * cond + 1e-300)[fin].all())
    # not finite alike (within a rounding of the largest FP64 value either side may still be finite)
    bad = ~torch.isfinite(ref)
    assert bool((~torch.isfinite(chi2[bad]) | (chi2[bad] > 1e308)).all())


# A and B of one size, so that their quotients are ordinary
@pytest.mark.parametrize("size,sigma", [(1e-290, 1e-100), (1e-290, 1e100), (1e290, 1e-100), (1e290, 1e100), (1.0, 1e-100),
                                        (1e-250, 0.1), (1e-307, 0.1), (1e307, 0.1)])
@pytest.mark.parametrize("n", [70, 5500])  # (5500: written in rank order through bins)
def test_values_and_errors_of_extreme_size(ctx, size, sigma, n):
    import microsn_gb300 as mlc
    rng = np.random.default_rng(n)
    A, B = (torch.as_tensor(np.exp(rng.uniform(-1, 1, (n, 3))) * size, device=DEV) for _ in range(2))
    dA, dB = torch.diff(A, dim=1).contiguous(), torch.diff(B, dim=1).contiguous()
    # only epochs with a value on both sides: a 1 against 1e-290 is no ordinary quotient
    v = mlc.Chi2Vars(2, np.array([0, 1], np.int32), np.array([1, 0], np.int32), np.array([0.3, 0.6]), np.array([0.2, 0.9]),
                     np.array([0.7, 1.2]), np.array([sigma, 2 * sigma]), 0.0)
    edges = mlc.bin_edges(40, 1e-2, 1e2)
    rank, lower, nper = mlc.setup_integral(ctx, A, B, edges)
    ref, cond = _reference(v, A, dA, B, dB)
    _check(mlc.calculate_chi2(ctx, v, A, dA, B, dB), ref.reshape(-1), cond.reshape(-1))
    at = rank.to(torch.int64) & 0xFFFFFFFF
    ranked = mlc.calculate_chi2(ctx, v, A, dA, B, dB, rank)
    _check(ranked[at], ref.reshape(-1), cond.reshape(-1))
    fc, _, fn = mlc.pair_bin_fused(ctx, v, A, dA, B, dB, edges)
    assert np.array_equal(fn, nper)
    for i in np.nonzero(nper)[0]:
        mean = ranked[int(lower[i]):int(lower[i]) + int(nper[i])].mean().item()
        assert abs(fc[i] - mean) <= 1e-12 * mean


# every location of its own size, 1e-150 to 1e150: some squares overflow, the others are compared
@pytest.mark.parametrize("n", [300, 1100])
def test_curves_of_all_sizes(ctx, n):
    import microsn_gb300 as mlc
    rng = np.random.default_rng(n)
    A, B = (torch.as_tensor(np.exp(rng.normal(0, 1, (n, 3))) * 10.0 ** rng.integers(-150, 150, (n, 1)), device=DEV)
            for _ in range(2))
    dA, dB = torch.diff(A, dim=1).contiguous(), torch.diff(B, dim=1).contiguous()
    v = _vars([0.7, 1.2, 1.1], [0.1, 0.15, 0.3])
    ref, cond = _reference(v, A, dA, B, dB)
    assert 0.2 < torch.isfinite(ref).double().mean().item() < 1
    _check(mlc.calculate_chi2(ctx, v, A, dA, B, dB), ref.reshape(-1), cond.reshape(-1))
