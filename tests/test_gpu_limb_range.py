"""FP64 convolutions at the upper end of the exponent range: sums beyond it come out as infinities
or NaN, never as finite values."""
import numpy as np
import pytest

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
