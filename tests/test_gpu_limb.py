"""Transforms in fixed-grid limbs (csrc/limb.cuh) against the FP64 oracle: every row length and
column split with a limb kernel, profiles narrower and wider than one column block, and
values at the ends of the FP64 and FP32 exponent ranges."""
import numpy as np
import pytest

import oracle
from microsn_gb300 import synth

pytestmark = pytest.mark.gpu

# (Nx, Ny): Nx/2 = 1000, 2000, 4096, 5000 points per row; Ny = N1 x N2 of 40x40, 40x50, 50x50,
# 64x64, 50x80, 80x80, 100x100, 128x128; 2400 (48x50) and 2160 rows (45x48) mix limb and generic passes
SIZES = [(2000, 1600), (2000, 2000), (4000, 2500), (8192, 4096), (10000, 4000), (2000, 6400), (2000, 10000),
         (2000, 16384), (4000, 2400), (2000, 2160)]


def _map(Nx, Ny, seed):
    rng = np.random.default_rng(seed)
    m = np.exp(rng.standard_normal((Ny, Nx)) * 0.8)
    m[Ny // 3] = 0.0  # a row of zeros
    m[Ny // 2, Nx // 2] = 300.0
    return m


def _check(got, ref, prec, Nx, Ny):
    rms = np.sqrt(np.mean(ref * ref))
    err = np.abs(got.astype(np.float64) - ref)
    if prec == "f64":
        # every pass rounds to 2^-53; numpy's own transform is within a few 2^-53 log2 N norm-wise
        assert err.max() <= 16 * 2.0 ** -53 * np.log2(Nx * Ny) * rms
    else:
        # the pixel's own rounding (half an ulp) plus 2^-46 S per pass, S below 2^10 rms
        assert np.max(err - (1 + 2.0 ** -10) * 2.0 ** -24 * np.abs(ref)) <= 2.0 ** -34 * rms


@pytest.mark.parametrize("Nx,Ny", SIZES)
@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_limb_convolution_matches_oracle(ctx, Nx, Ny, prec):
    import microsn_gb300 as mlc
    mp = _map(Nx, Ny, Nx + Ny)
    if prec == "f32":
        mp = mp.astype(np.float32)
    m = mlc.Map(ctx, mp, prec)
    if prec == "f32":
        m.set_fft("f32x2")
    # 12 and 122 rows: half widths 6 and 61, the second wider than the 40- and 50-row blocks
    for p in (mlc.profile("gaussian", 3.0, 1.0, ref_compat=False), mlc.profile("exponential", 30.5, 1.0, ref_compat=False)):
        got = mlc.convolve(ctx, m, p).cpu().numpy()
        ref = oracle.conv_fft_workers(mp.astype(np.float64), mlc.profile_raster(p))
        _check(got, ref, prec, Nx, Ny)
    m.close()


@pytest.mark.parametrize("prec,scale", [("f64", 1e250), ("f64", 1e-250), ("f32", 1e25), ("f32", 1e-18)])
def test_limb_convolution_scales_with_the_map(ctx, prec, scale):
    import microsn_gb300 as mlc
    Nx, Ny = 2000, 2000
    mp = _map(Nx, Ny, 5) * scale
    if prec == "f32":
        mp = mp.astype(np.float32)
    m = mlc.Map(ctx, mp, prec)
    if prec == "f32":
        m.set_fft("f32x2")
    p = mlc.profile("gaussian", 3.0, 1.0, ref_compat=False)
    got = mlc.convolve(ctx, m, p).cpu().numpy().astype(np.float64) / scale
    ref = oracle.conv_fft_workers(mp.astype(np.float64) / scale, mlc.profile_raster(p))
    rms = np.sqrt(np.mean(ref * ref))
    # (one more rounding for the division)
    tol = 17 * 2.0 ** -53 * np.log2(Nx * Ny) * rms if prec == "f64" else 2.0 ** -24 * 1.01 * np.abs(ref) + 2.0 ** -34 * rms
    assert np.all(np.abs(got - ref) <= tol)
    m.close()


@pytest.mark.parametrize("prec", ["f64", "f32"])
def test_limb_convolution_of_zeros_and_of_a_nan(ctx, prec):
    import microsn_gb300 as mlc
    N = 2000
    mp = np.zeros((N, N), np.float64 if prec == "f64" else np.float32)
    p = mlc.profile("gaussian", 3.0, 1.0, ref_compat=False)
    for fill, want in ((0.0, 0.0), (np.nan, np.nan)):
        mp[7, 9] = fill
        m = mlc.Map(ctx, mp, prec)
        if prec == "f32":
            m.set_fft("f32x2")
        got = mlc.convolve(ctx, m, p).cpu().numpy()
        assert np.array_equal(got, np.full_like(got, want), equal_nan=True)
        m.close()
