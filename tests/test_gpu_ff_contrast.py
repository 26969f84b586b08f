"""FP32 maps with float-float transforms keep their faint pixels: on maps whose pixels span six
to nine orders of magnitude every convolved pixel is the FP64 one rounded to FP32, up to the
float-float error of its transforms."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _map(Ny, Nx, sd, seed):
    """exp of a Gaussian field that is smooth over a few pixels, mean 1."""
    g = torch.randn((Ny, Nx), generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV, dtype=torch.float64)
    f = torch.fft.rfft2(g)
    ky, kx = torch.fft.fftfreq(Ny, device=DEV)[:, None], torch.fft.rfftfreq(Nx, device=DEV)[None, :]
    g = torch.fft.irfft2(f / (1.0 + (kx * kx + ky * ky) * 4000.0), s=(Ny, Nx))
    m = torch.exp(sd * (g - g.mean()) / g.std())
    return (m / m.mean()).float().contiguous()


def _convolved(m, prof):
    Ny, Nx = m.shape
    N = prof.shape[0]
    k = torch.zeros((Ny, Nx), dtype=torch.float64, device=DEV)
    at = torch.arange(N, device=DEV) - N // 2
    k[(at % Ny)[:, None], (at % Nx)[None, :]] = torch.as_tensor(prof, device=DEV)
    return torch.fft.irfft2(torch.fft.rfft2(m.double()) * torch.fft.rfft2(k), s=(Ny, Nx))


def _excess(got, ref):
    """Error beyond the pixel's own rounding (half an ulp), against the rms of the map and of the pixel's row."""
    over = (got.double() - ref).abs() - 2.0 ** -24 * (1 + 2.0 ** -10) * ref.abs()
    sq = ref.square()
    return (over / (sq.mean().sqrt() + sq.mean(1, keepdim=True).sqrt())).max().item()


# A float-float operation is within a few 2^-47 of its operands.  The last pass's gather, over some
# five levels, to about 2^-46 of the row's rms (a row with a bright pixel has a larger one than
# the map), those of the passes before it to about 2^-46 of the map's; the largest of 10^8
# pixels is six of those or so: 2^-42 leaves a factor of two.  torch's FP64 is at 2^-50.
LIMIT = 2.0 ** -42

# rows of 1000, 1500, 2000, 4096 and 5000 points; columns 40 x 50, 48 x 50, 50 x 60, 50 x 80, 64 x 64
SIZES = [(2000, 2000), (2000, 3000), (2400, 4000), (4096, 8192), (4000, 10000), (3000, 810)]


@pytest.mark.parametrize("Ny,Nx", SIZES)
@pytest.mark.parametrize("sd", [0.8, 2.0])
def test_faint_pixels_of_fp32_maps(ctx, Ny, Nx, sd):
    import microsn_gb300 as mlc
    mp = _map(Ny, Nx, sd, Nx + Ny)
    m = mlc.Map(ctx, mp, "f32")
    m.set_fft("f32x2")
    for p in (mlc.profile("uniform", 1.0, 1.0, ref_compat=False), mlc.profile("exponential", 8.0, 1.0, ref_compat=False)):
        ref = _convolved(mp, mlc.profile_raster(p))
        assert _excess(mlc.convolve(ctx, m, p), ref) <= LIMIT
    m.close()


def test_faint_pixels_from_cached_spectra(ctx):
    """mlc_convolve_many keeps its profiles' spectra (here at 2000 x 10000, N2 = 100): the first call, which
    makes them, and the second, which starts from them."""
    import microsn_gb300 as mlc
    mp = _map(10000, 2000, 2.0, 7)
    m = mlc.Map(ctx, mp, "f32")
    m.set_fft("f32x2")
    profs = [mlc.profile("uniform", 1.0, 1.0, ref_compat=False), mlc.profile("exponential", 8.0, 1.0, ref_compat=False)]
    refs = [_convolved(mp, mlc.profile_raster(p)) for p in profs]
    for _ in range(2):
        out = mlc.convolve_many(ctx, m, profs)
        for k, ref in enumerate(refs):
            assert _excess(out[k], ref) <= LIMIT
    m.close()


@pytest.mark.parametrize("N", [2000, 4000, 10000])
def test_fp64_pixels_cost_their_bytes(ctx, N):
    """The last pass of a float-float convolution into FP64 pixels against FP32 ones: twice the pixels'
    bytes and the conversions on the FP64 pipe, which all warps share, are less than twice the time."""
    import microsn_gb300 as mlc
    p = mlc.profile("exponential", 16.0, 1.0, ref_compat=False)
    ms = []
    ctx.set_timing(True)
    try:
        for prec, dt in (("f32", torch.float32), ("f64", torch.float64)):
            m = mlc.Map(ctx, torch.rand((N, N), dtype=dt, device=DEV) + 0.5, prec)
            m.set_fft("f32x2")
            out = mlc.convolve(ctx, m, p)
            times = []
            for _ in range(7):
                ctx.kernel_times()
                mlc.convolve(ctx, m, p, out=out)
                times.append(ctx.kernel_times()["fft_rows_c2r"][0])
            ms.append(sorted(times)[3])
            m.close()
    finally:
        ctx.set_timing(False)
    assert ms[1] <= 1.75 * ms[0]
