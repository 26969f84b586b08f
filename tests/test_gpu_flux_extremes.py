"""The flux-ratio likelihood of magnifications near the ends of FP32, on both sides of the size from
which its terms are scaled: the chi2 of the undivided terms."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("N", [200, 3300])
@pytest.mark.parametrize("size,df", [(2.0 ** -118, 2.0 ** -14), (2.0 ** -118, 2.0 ** 14), (2.0 ** 118, 2.0 ** -14),
                                     (2.0 ** 118, 2.0 ** 14), (1.0, 0.25)])
def test_magnifications_of_extreme_size(ctx, N, size, df):
    import microsn_gb300 as mlc
    F, T = 2, 9
    rng = np.random.default_rng(N)
    fo = rng.uniform(0.6, 1.4, (F, T)).astype(np.float32)
    dfo = (rng.uniform(0.6, 1.0, (F, T)) * df).astype(np.float32)
    g = torch.Generator(device=DEV).manual_seed(N)
    m1, m2 = (torch.exp(0.3 * torch.randn((N, F, T), generator=g, device=DEV)) * size for _ in range(2))
    like, chi2 = mlc.flux_ratio_chi2(ctx, fo, dfo, m1, m2, want_chi2=True)
    ref = torch.zeros((N, N), dtype=torch.float64, device=DEV)
    tol = torch.zeros_like(ref)
    a, b = m1.reshape(N, -1).double(), m2.reshape(N, -1).double()
    for k, (f, d) in enumerate(zip(fo.reshape(-1).astype(np.float64), dfo.reshape(-1).astype(np.float64))):
        q = a[:, k][None, :] / b[:, k][:, None]
        t = (f - q) / d
        ref += 0.5 * t * t
        # 1/mu2 or B, and t, each rounded to 2^-24 of its size; the sum's own rounding below
        tol += t.abs() * (2 * q + abs(f)) / d * 2.0 ** -24 + 2 * t * t * 2.0 ** -24
    tol += F * T * 2.0 ** -24 * ref
    assert bool(((chi2.double() - ref).abs() <= tol).all())
    want = torch.exp(-chi2.double()).sum().item()
    assert abs(like - want) <= 1e-6 * want + 1e-300
