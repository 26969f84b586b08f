"""Limb transforms of lengths without an unrolled kernel (csrc/fft_limb_any.cu) against the FP64
oracle: every radix first and last, odd lengths, rows and columns of one level, the widest
rows that fit, and sizes that no transform takes."""
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
    (15000, 2592),  # 7500 (10 10 5 5 3), 48 x 54; these rows end at 13000
    (12500, 128),   # 6250 (10 5 5 5 5), 8 x 16
    (26, 48),       # 13: no transform of this length
    (64, 32),       # 32 (8 4), 4 x 8
    (36, 250),      # 18 (9 2), 10 x 25
    (36, 125),      # odd
    (108, 1500),    # 54 (9 6); two limbs take more than four rows per SM
    (64, 2048),     # 32 (8 4)
    (36, 1000),     # 18 (9 2)
    (20, 1080),     # 10: one level
    (9216, 1024),   # 4608 (9 8 8 8)
]


@pytest.mark.parametrize("Nx,Ny", SIZES)
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_convolution_matches_oracle(ctx, Nx, Ny, prec):
    import microsn_gb300 as mlc
    rng = np.random.default_rng(Nx * Ny)
    mp = np.exp(rng.standard_normal((Ny, Nx)) * 0.8)
    mp[Ny // 3] = 0.0
    mp[Ny // 2, Nx // 2] = 300.0
    if prec == "f32":
        mp = mp.astype(np.float32)
    if Nx > 13000 or Nx == 26 or Ny % 2:  # refused, as documented
        with pytest.raises(mlc.MlcError):
            m = mlc.Map(ctx, mp, prec)
            m.set_fft("native" if prec == "f64" else "f32x2")
            mlc.convolve(ctx, m, mlc.profile("gaussian", 3.0, 1.0, ref_compat=False))
        return
    m = mlc.Map(ctx, mp, prec)
    if prec == "f32":
        m.set_fft("f32x2")
    profs = [mlc.profile("gaussian", 3.0, 1.0, ref_compat=False)]
    if min(Nx, Ny) > 400:  # wider than a column block
        profs.append(mlc.profile("exponential", 30.5, 1.0, ref_compat=False))
    for p in profs:
        got = mlc.convolve(ctx, m, p).cpu().numpy().astype(np.float64)
        ref = oracle.conv_fft_workers(mp.astype(np.float64), mlc.profile_raster(p))
        rms = np.sqrt(np.mean(ref * ref))
        if prec == "f64":  # every pass rounds to 2^-53; numpy's transform is within a few 2^-53 log2 N
            tol = 16 * 2.0 ** -53 * np.log2(Nx * Ny) * rms
        else:  # the pixel's own rounding, plus 2^-46 S per pass with S below 2^10 rms
            tol = (1 + 2.0 ** -10) * 2.0 ** -24 * np.abs(ref) + 2.0 ** -34 * rms
        assert np.all(np.abs(got - ref) <= tol)
    m.close()


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_convolution_of_a_nan_is_nan(ctx, prec):
    import microsn_gb300 as mlc
    mp = np.zeros((150, 108), np.float64 if prec == "f64" else np.float32)
    p = mlc.profile("gaussian", 3.0, 1.0, ref_compat=False)
    for fill, want in ((0.0, 0.0), (np.nan, np.nan)):
        mp[7, 9] = fill
        m = mlc.Map(ctx, mp, prec)
        if prec == "f32":
            m.set_fft("f32x2")
        got = mlc.convolve(ctx, m, p).cpu().numpy()
        assert np.array_equal(got, np.full_like(got, want), equal_nan=True)
        m.close()
