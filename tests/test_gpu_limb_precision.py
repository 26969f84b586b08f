"""FP64 transforms in limbs are as exact as FP64 arithmetic: rms and faintest pixels of maps of
ordinary and of high contrast, every kind of row length, against exactly rounded sums."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _map(Ny, Nx, sd, seed):
    g = torch.randn((Ny, Nx), generator=torch.Generator(device=DEV).manual_seed(seed), device=DEV, dtype=torch.float64)
    f = torch.fft.rfft2(g)
    ky, kx = torch.fft.fftfreq(Ny, device=DEV)[:, None], torch.fft.rfftfreq(Nx, device=DEV)[None, :]
    g = torch.fft.irfft2(f / (1.0 + (kx * kx + ky * ky) * 4000.0), s=(Ny, Nx))
    m = torch.exp(sd * (g - g.mean()) / g.std())
    return (m / m.mean()).contiguous()


# rows of 600, 1000, 1500, 2000, 3000, 4096 and 5000 points, by run-time radices and unrolled
@pytest.mark.parametrize("Ny,Nx", [(1200, 1200), (2000, 2000), (2000, 3000), (4000, 4000), (3000, 6000), (4096, 8192),
                                   (10000, 10000)])
@pytest.mark.parametrize("sd", [0.8, 2.0])
def test_fp64_convolution_keeps_fp64_precision(ctx, Ny, Nx, sd):
    import microsn_gb300 as mlc
    mp = _map(Ny, Nx, sd, Nx + 7)
    mh = mp.cpu().numpy()
    m = mlc.Map(ctx, mp, "f64")
    prof = mlc.profile("uniform", 1.0, 1.0, ref_compat=False)
    raster = mlc.profile_raster(prof)
    h = raster.shape[0] // 2
    got = mlc.convolve(ctx, m, prof).reshape(-1)
    m.close()
    at = torch.cat([torch.topk(got, 200, largest=False).indices,
                    torch.randint(0, Ny * Nx, (400,), generator=torch.Generator(device=DEV).manual_seed(1), device=DEV)])
    off = np.arange(raster.shape[0]) - h
    err = []
    for q, v in zip(at.tolist(), got[at].tolist()):
        y, x = divmod(q, Nx)
        w = mh[np.ix_((y - off) % Ny, (x - off) % Nx)]
        err.append(v - float((raster.astype(np.longdouble) * w.astype(np.longdouble)).sum()))
    rms = got.square().mean().sqrt().item()
    err = np.abs(err) / rms
    # Six passes of FP64 arithmetic, each 2^-53 times about the square root of log2 of its length
    # over 2 (random roundings of one in two butterflies): 2^-53 sqrt(2 (12 + 13 + 13) / 2) = 2^-50.4
    # of the rms; the maximum of 600 pixels within four of those.
    assert math.sqrt(np.mean(err[:200] ** 2)) <= 2.0 ** -50.4
    assert math.sqrt(np.mean(err[200:] ** 2)) <= 2.0 ** -50.4
