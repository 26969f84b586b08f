"""FP32 and float-float transforms of lengths without an unrolled kernel (csrc/fft_any_real.cuh)
against the FP64 oracle: every radix, two to five levels, lengths of one level (which keep
the general kernel), and a row too long for both buffers of the forward pass."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

# Nx/2 points per row (radices), Ny = N1 x N2
SIZES = [
    (6000, 3000),   # 3000 (10 10 10 3), 50 x 60
    (108, 150),     # 54 (9 6), 10 x 15
    (1000, 1080),   # 500 (10 10 5), 30 x 36
    (3000, 4860),   # 1500 (10 10 5 3), 60 x 81
    (9216, 512),    # 4608 (9 8 8 8), 16 x 32
    (6250, 1250),   # 3125 (5 5 5 5 5), 25 x 50
    (64, 32),       # 32 (8 4), 4 x 8
    (20, 36),       # 10: one level; 6 x 6
    (36, 250),      # 18 (9 2), 10 x 25
    (24000, 96),    # 12000 (10 10 10 4 3), FP32 only: rows in float-float end at 13000
    (25600, 48),    # 12800 (10 10 8 8 2), FP32 only
    # (fewer rows than six per SM keep the general kernel)
    (108, 1500),    # 54 (9 6)
    (64, 2048),     # 32 (8 4)
    (36, 1000),     # 18 (9 2)
    (20, 1080),     # 10: one level
    (9216, 1024),   # 4608 (9 8 8 8)
    (24000, 960),   # 12000, FP32 only
]


@pytest.mark.parametrize("Nx,Ny", SIZES)
@pytest.mark.parametrize("prec", ["f32", "f64"])
def test_convolution_matches_oracle(ctx, Nx, Ny, prec):
    import microsn_gb300 as mlc
    if prec == "f64" and Nx > 13000:
        pytest.skip("FP32 only")
    rng = np.random.default_rng(Nx * Ny + 1)
    mp = np.exp(rng.standard_normal((Ny, Nx)) * 0.8)
    mp[Ny // 3] = 0.0
    mp[Ny // 2, Nx // 2] = 300.0
    if prec == "f32":
        mp = mp.astype(np.float32)
    m = mlc.Map(ctx, mp, prec)
    m.set_fft("native" if prec == "f32" else "f32x2")
    # every pass adds a few units of the arithmetic (2^-24; float-float at least 2^-44) of the
    # rms of what it transforms: the map going in, no more than that coming out
    tol = 16 * (2.0 ** -24 if prec == "f32" else 2.0 ** -44) * np.log2(Nx * Ny)
    rms = np.sqrt(np.mean(mp.astype(np.float64) ** 2))
    profs = [mlc.profile("gaussian", 2.0, 1.0, ref_compat=False)]
    if min(Nx, Ny) > 400:  # wider than a column block
        profs.append(mlc.profile("exponential", 30.5, 1.0, ref_compat=False))
    for p in profs:
        got = mlc.convolve(ctx, m, p).cpu().numpy().astype(np.float64)
        ref = oracle.conv_fft_workers(mp.astype(np.float64), mlc.profile_raster(p))
        assert np.max(np.abs(got - ref)) <= tol * rms
    m.close()
