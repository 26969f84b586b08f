"""The flux-ratio likelihood across its two tile forms: sizes around the form's limit, ragged
tiles and chunks, zero and extreme observations, against FP64 sums on the device."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,F,T,case", [(1, 1, 1, ""), (65, 2, 17, "zero flux"), (300, 2, 5, "tiny df"), (3000, 1, 3, ""),
                                        (3073, 1, 16, ""), (3201, 1, 17, "zero flux"), (3333, 3, 11, "tiny df")])
def test_flux_ratio_tiles(ctx, N, F, T, case):
    import microsn_gb300 as mlc
    rng = np.random.default_rng(N)
    fo = rng.uniform(0.6, 1.4, (F, T)).astype(np.float32)
    dfo = rng.uniform(0.2, 0.6, (F, T)).astype(np.float32)
    if case == "zero flux":
        fo[0, :2] = 0.0
    elif case == "tiny df":  # beyond the scaled terms' range: they stay unscaled
        dfo[0, 0] = 1e-6
    g = torch.Generator(device="cuda:0").manual_seed(N)
    m1, m2 = (torch.exp(0.4 * torch.randn((N, F, T), generator=g, device="cuda:0")) for _ in range(2))
    like, chi2 = mlc.flux_ratio_chi2(ctx, fo, dfo, m1, m2, want_chi2=True)
    ref = torch.zeros((N, N), dtype=torch.float64, device="cuda:0")
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
