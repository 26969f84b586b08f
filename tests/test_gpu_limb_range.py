"""FP64 convolutions at the ends of the exponent range: sums beyond it come out as infinities or
NaN, never as finite values, and values near and below its lower end keep what FP64 has there."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

# unrolled rows and columns; run-time radices for both; unrolled rows with run-time columns
SIZES = [(2000, 2000), (1500, 1500), (2000, 2160)]


def _map(Ny, Nx):
    rng = np.random.default_rng(Nx)
    return np.exp(0.8 * rng.standard_normal((Ny, Nx)))


@pytest.mark.parametrize("Nx,Ny", SIZES)
@pytest.mark.parametrize("scale", [1e303, 1e306])  # sums up to 2^7 and 2^17 times the largest FP64 value
def test_sums_beyond_fp64_are_not_finite(ctx, Nx, Ny, scale):
    import microsn_gb300 as mlc
    m = mlc.Map(ctx, _map(Ny, Nx) * scale, "f64")
    got = mlc.convolve(ctx, m, mlc.profile("gaussian", 3.0, 1.0, ref_compat=False)).cpu().numpy()
    m.close()
    assert not np.isfinite(got).any()


@pytest.mark.parametrize("Nx,Ny", SIZES)
@pytest.mark.parametrize("exponent", [-970, -1000, -1040])  # (the last one: subnormal pixels)
def test_small_values_keep_fp64_precision(ctx, Nx, Ny, exponent):
    import microsn_gb300 as mlc
    mp = np.ldexp(_map(Ny, Nx), exponent)
    p = mlc.profile("gaussian", 3.0, 1.0, ref_compat=False)
    m = mlc.Map(ctx, mp, "f64")
    got = np.ldexp(mlc.convolve(ctx, m, p).cpu().numpy(), -exponent)
    m.close()
    ref = oracle.conv_fft_workers(np.ldexp(mp, -exponent), mlc.profile_raster(p))
    rms = np.sqrt(np.mean(ref * ref))
    # every pass rounds to 2^-53, or to half of 2^-1074: the first column pass does so on the Nx Ny
    # values that a pixel is the sum of, sqrt(2 Nx Ny / 3) of them as a random walk, times six
    # for the largest pixel
    tol = 16 * 2.0 ** -53 * np.log2(Nx * Ny) * rms + 6 * np.sqrt(2 * Nx * Ny / 3) * 2.0 ** (-1075 - exponent)
    assert np.abs(got - ref).max() <= tol
