"""The work whose speed is followed: one case per kind of call that a program makes of this
package, over the range of sizes, data types and options that the calls are used at.

A case is a dict of plain values with its kind in "kind".  prepare() makes what the program
has in hand before the call (maps, tracks, curves; one context for the whole process), run()
makes the call through the package's public functions and returns everything it computes,
exact() restates the same results in 64 bits with torch and numpy alone.
"""
import math

import numpy as np
import torch

import microsn_gb300 as mlc

DEV = "cuda:0"
RHALF_PX = (2, 4, 8, 16, 32, 48, 64, 96)   # half-light radii of the batched step
SEASONS, SEASON_LEN, GAP = 3, 120.0, 245.0  # observing seasons in days
WIDTH = 20.0                                # map side in Einstein radii
RATIO_SIZES = (0.0, 0.05, 0.1, 0.2, 0.3)    # expanding source, Einstein radii
RATIO_DATA = ((0.7, 1.2, 1.4, 1.1, 0.9), (5.0, 7.0, 12.0, 14.0, 17.0), (0.1, 0.15, 0.1, 0.1, 0.15))
FIT_RADII = tuple(float(r) for r in np.geomspace(4.0, 32.0, 16))


def listed():
    return [
        # The batched workload at full size: new pixels of a 10000^2 FP32 map, 16 profiles,
        # 10^6 seasonal tracks, float-float transforms, magnitudes on the device.
        dict(name="step_10000_f32x2", kind="step", n=10000, prec="f32", fft="f32x2", nprof=16, ntracks=1_000_000,
             host=False),
        # The same step of a double-precision run (the default for FP64 maps) at an ordinary size.
        dict(name="step_4000_f64", kind="step", n=4000, prec="f64", fft="native", nprof=4, ntracks=50_000, host=False),
        # A program that keeps its arrays on the host: pixels and tracks up, light curves down;
        # a map side without a register row kernel, FP32 throughout.
        dict(name="step_3000_f32_host", kind="step", n=3000, prec="f32", fft="native", nprof=3, ntracks=20_000,
             host=True),
        # The small double-precision end-to-end run: one Gaussian, 10^4 tracks x 50 epochs,
        # offset chi2, sort and histogram.
        dict(name="target_2000_f64", kind="target", n=2000, fft="native", ntracks=10_000, epochs=50),
        # The reference driver's light curves: fixed locations, expanding Gaussian source, FP64.
        dict(name="expanding_10000_f64", kind="expanding", n=10000, nsizes=5, nloc=9216),
        # A supernova's convolutions: limb-darkened discs of growing radius in three bands.
        dict(name="many_8192_f32", kind="many", n=8192, prec="f32", fft="native", nprof=12, rmax=100.0),
        # One convolution of a new map, at a size that no register kernel covers.
        dict(name="single_6000_f32", kind="many", n=6000, prec="f32", fft="native", nprof=1, rmax=24.0),
        # The reference's pair path: z rank of all pairs, ratio chi2 in rank order, bin means.
        dict(name="ratio_ranked_9216", kind="ratio", nloc=9216, fused=False, nbins=300),
        # The same statistic without the rank, as a likelihood scan calls it.
        dict(name="ratio_fused_9216", kind="ratio", nloc=9216, fused=True, nbins=300),
        # Magnitude-difference chi2 of all pairs of two images' curves, histogram and best pairs.
        dict(name="magdiff_100000", kind="magdiff", na=100_000, nb=100_000, epochs=128, k=10_000, matrix=False),
        # One iteration of the gradient fit: chi2 and its gradient for 4096 tracks x 80 epochs.
        dict(name="fit_4096", kind="fit", n=4000, ntracks=4096, epochs=80),
        # The multi-filter flux-ratio likelihood of all location pairs.
        dict(name="flux_10000", kind="flux", nloc=10_000, filters=7, epochs=10),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    """A map side the transforms take (even, factors 2, 3 and 5), over the logarithm of the range."""
    want = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    smooth = [2 ** a * 3 ** b * 5 ** c for a in range(1, 15) for b in range(9) for c in range(7)]
    return min((s for s in smooth if lo <= s <= hi), key=lambda s: abs(math.log(s / want)))


def draw(rng):
    kind = rng.choice(("step", "step", "target", "expanding", "many", "ratio", "magdiff", "fit", "flux"))
    if kind == "step":
        prec, fft = rng.choice((("f32", "f32x2"), ("f32", "native"), ("f64", "native"), ("f64", "f32x2")))
        top = 10000 if prec == "f32" else 4096
        host = rng.random() < 0.25
        return dict(kind=kind, n=_side(rng, 500, 3000 if host else top), prec=prec, fft=fft, nprof=rng.randint(1, 16),
                    ntracks=_log_uniform(rng, 200, 20_000 if host else 300_000), host=host)
    if kind == "target":
        return dict(kind=kind, n=_side(rng, 500, 4000), fft=rng.choice(("native", "f32x2")),
                    ntracks=_log_uniform(rng, 100, 50_000), epochs=rng.randint(20, 128))
    if kind == "expanding":
        return dict(kind=kind, n=_side(rng, 1000, 6000), nsizes=rng.randint(2, 5), nloc=_log_uniform(rng, 100, 20_000))
    if kind == "many":
        prec, fft = rng.choice((("f32", "native"), ("f32", "f32x2"), ("f64", "native"), ("f64", "f32x2")))
        return dict(kind=kind, n=_side(rng, 500, 8192 if prec == "f32" else 4096), prec=prec, fft=fft,
                    nprof=rng.randint(1, 8), rmax=float(rng.randint(4, 100)))
    if kind == "ratio":
        return dict(kind=kind, nloc=_log_uniform(rng, 300, 9216), fused=rng.random() < 0.5, nbins=rng.randint(50, 500))
    if kind == "magdiff":
        return dict(kind=kind, na=_log_uniform(rng, 300, 100_000), nb=_log_uniform(rng, 300, 60_000),
                    epochs=rng.randint(20, 128), k=rng.randint(10, 5000), matrix=False)
    if kind == "fit":
        return dict(kind=kind, n=_side(rng, 1000, 4000), ntracks=_log_uniform(rng, 64, 20_000),
                    epochs=rng.randint(20, 200))
    return dict(kind=kind, nloc=_log_uniform(rng, 300, 10_000), filters=rng.randint(2, 8), epochs=rng.randint(5, 40))


# ----------------------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _map(n, seed, dtype):
    """A positive, heavy-tailed map of mean 1 with structure from a few pixels up, as ray-shot
    magnification maps have: the exponential of a Gaussian field with a steep spectrum."""
    g = torch.randn((n, n), generator=_gen(seed), device=DEV, dtype=torch.float32)
    f = torch.fft.rfft2(g)
    ky = torch.fft.fftfreq(n, device=DEV)[:, None]
    kx = torch.fft.rfftfreq(n, device=DEV)[None, :]
    f *= 1.0 / (1.0 + (kx * kx + ky * ky) * 4000.0)
    g = torch.fft.irfft2(f, s=(n, n))
    del f
    g = (g - g.mean()) / g.std()
    m = torch.exp(0.8 * g)
    m = m / m.mean()
    return m.to(dtype).contiguous()


def _uniform(g, n):
    return torch.rand(n, generator=g, device=DEV, dtype=torch.float64)


def _starts(g, n, margin, phi, length, ntracks):
    """Start coordinates that keep straight tracks of the given lengths inside the map."""
    out = []
    for c in (torch.cos(phi), torch.sin(phi)):
        lo = margin + torch.clamp(-length * c, min=0)
        hi = n - margin - torch.clamp(length * c, min=0)
        out.append(lo + (hi - lo) * _uniform(g, ntracks))
    return out


def _tracks(n, ntracks, seed, dtype):
    """Straight tracks with U{20..200} epochs in three seasons, speeds in pixels per day."""
    g = _gen(seed + 7777)
    # (the counts are one fixed draw in another order, so that every seed has as many epochs)
    cnt = torch.randint(20, 201, (ntracks,), generator=_gen(1), device=DEV)
    cnt = cnt[torch.randperm(ntracks, generator=g, device=DEV)]
    off = torch.zeros(ntracks + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(cnt, 0)
    tid = torch.repeat_interleave(torch.arange(ntracks, device=DEV), cnt)
    j = torch.arange(int(off[-1]), device=DEV) - off[tid]
    nk = cnt[tid]
    season = (j * SEASONS) // nk
    first = (season * nk + SEASONS - 1) // SEASONS
    ns = ((season + 1) * nk + SEASONS - 1) // SEASONS - first
    t = season.double() * (SEASON_LEN + GAP) + ((j - first).double() + _uniform(g, j.numel())) / ns * SEASON_LEN
    del tid, j, nk, season, first, ns
    phi = _uniform(g, ntracks) * (2 * math.pi)
    v = 0.05 + 0.95 * _uniform(g, ntracks)
    tmax = t[off[1:] - 1]
    margin = min(2.0 * RHALF_PX[-1] + 2, n / 8.0)
    room = 0.9 * (n - 2 * margin)
    v = torch.where(v * tmax > room, room / tmax.clamp(min=1e-300), v)
    x0, y0 = _starts(g, n, margin, phi, v * tmax, ntracks)
    tr = dict(x0=x0, y0=y0, phi=phi, v=v, off=off, t=t)
    return {k: (a if k == "off" else a.to(dtype)) for k, a in tr.items()}


def _step_profiles(nprof, n):
    """(shape, half-light radius in pixels) of the batched step's profiles, as many as asked."""
    radii = [r for r in RHALF_PX if 4 * r <= n // 2]
    every = [(s, float(r)) for s in ("uniform", "exponential") for r in radii]
    return [every[(k * len(every)) // nprof if nprof <= len(every) else k % len(every)] for k in range(nprof)]


def _limb_profiles(nprof, rmax):
    """(radius, limb darkening) of a photosphere that grows to rmax pixels, three bands an epoch."""
    radii = np.linspace(1.0, rmax, max(2, -(-nprof // 3))) if nprof > 1 else [rmax]
    return [(float(r), u) for r in radii for u in (0.6, 0.45, 0.3)][:nprof]


def _target_inputs(case, seed):
    n, k, T = case["n"], case["ntracks"], case["epochs"]
    g = _gen(seed + 99)
    phi = _uniform(g, k) * (2 * math.pi)
    speed = min(5.0, 0.8 * (n - 80.0) / (T - 1))
    x0, y0 = _starts(g, n, 40.0, phi, torch.full_like(phi, speed * (T - 1)), k)
    t = torch.arange(T, dtype=torch.float64, device=DEV)
    obs = 0.3 * torch.sin(t / 7.0) + 0.05 * torch.randn(T, generator=g, device=DEV, dtype=torch.float64)
    w = torch.full((T,), 1 / 0.05 ** 2, dtype=torch.float64, device=DEV)
    return _map(n, seed, torch.float64), (x0, y0, phi, torch.full_like(phi, speed)), t, obs, w


def _locations(case, seed):
    n = case["n"]
    margin = int(math.ceil(n / WIDTH * RATIO_SIZES[-1]))
    r = np.random.default_rng(seed)
    return [r.integers(margin, n - margin, case["nloc"]).astype(np.int32) for _ in range(2)]


def _ratio_inputs(case, seed):
    """Light curves of two images at every location: lognormal magnifications that smooth out
    as the source grows."""
    g = _gen(seed)
    out = []
    for _ in range(2):
        base = torch.randn((case["nloc"], 1), generator=g, device=DEV, dtype=torch.float64)
        step = torch.randn((case["nloc"], len(RATIO_SIZES)), generator=g, device=DEV, dtype=torch.float64)
        lc = torch.exp(0.7 * base + 0.15 * torch.cumsum(step, 1)).contiguous()
        out += [lc, (lc[:, 1:] - lc[:, :-1]).contiguous()]
    return out


def _curves(rows, T, g):
    """FP32 magnitude curves: a slow random walk about a level of its own."""
    x = torch.randn((rows, T), generator=g, device=DEV, dtype=torch.float32)
    x = torch.cumsum(x, 1) * (0.4 / math.sqrt(T))
    return (x + torch.randn((rows, 1), generator=g, device=DEV, dtype=torch.float32)).contiguous()


def _magdiff_inputs(case, seed):
    g = _gen(seed)
    T = case["epochs"]
    A, B = _curves(case["na"], T, g), _curves(case["nb"], T, g)
    w = 1.0 / np.random.default_rng(seed).uniform(0.02, 0.1, T) ** 2
    return A, B, w


def _fit_inputs(case, seed):
    n, k, T = case["n"], case["ntracks"], case["epochs"]
    g = _gen(seed + 5)
    t, _ = torch.sort(torch.randint(0, 3, (k, T), generator=g, device=DEV) * 365.0
                      + 150.0 * torch.rand((k, T), generator=g, device=DEV, dtype=torch.float64), dim=1)
    v = 0.02 + 0.06 * _uniform(g, k)
    phi = _uniform(g, k) * (2 * math.pi)
    x0, y0 = _starts(g, n, 80.0, phi, v * t[:, -1], k)
    R = 8.0 + 8.0 * _uniform(g, k)
    dm = 0.6 * _uniform(g, k) - 0.3
    theta = torch.stack([x0, y0, phi, v, R, dm], 1).float().contiguous()
    obs = (0.3 * torch.randn((k, 1), generator=g, device=DEV) + 0.1 * torch.randn((k, T), generator=g, device=DEV))
    w = torch.full((k * T,), 1 / 0.02 ** 2, device=DEV)
    off = torch.arange(k + 1, device=DEV, dtype=torch.int64) * T
    return theta, off, t.reshape(-1).float().contiguous(), obs.reshape(-1).float().contiguous(), w


def _flux_inputs(case, seed):
    r = np.random.default_rng(seed)
    F, T, N = case["filters"], case["epochs"], case["nloc"]
    fo = r.uniform(0.8, 1.2, (F, T)).astype(np.float32)
    dfo = r.uniform(0.05, 0.2, (F, T)).astype(np.float32)
    g = _gen(seed)
    mu = [torch.exp(0.3 * torch.randn((N, F, T), generator=g, device=DEV)).contiguous() for _ in range(2)]
    return fo, dfo, mu[0], mu[1]


_CTX = None


def _ctx():
    """The program's one context: workspaces, plans and tuned choices live as long as it does."""
    global _CTX
    if _CTX is None:
        _CTX = mlc.Context(0)
    return _CTX


def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    s = dict(case=case, ctx=ctx)
    if kind == "step":
        dt = torch.float64 if case["prec"] == "f64" else torch.float32
        pixels = _map(case["n"], seed, dt)
        s["map"] = mlc.Map(ctx, pixels, case["prec"])
        s["map"].set_fft(case["fft"])
        s["profiles"] = [mlc.profile(sh, r, 1.0, ref_compat=False) for sh, r in _step_profiles(case["nprof"], case["n"])]
        tr = _tracks(case["n"], case["ntracks"], seed, dt)
        if case["host"]:
            s["pixels"] = pixels.cpu().pin_memory()
            s["tracks"] = {k: a.cpu().pin_memory() for k, a in tr.items()}
            s["out"] = mlc.host_empty((case["nprof"], tr["t"].numel()), dt)
        else:
            s["pixels"], s["tracks"], s["out"] = pixels, tr, None
    elif kind == "target":
        mp, s["tracks"], s["t"], s["obs"], s["w"] = _target_inputs(case, seed)
        s["map"] = mlc.Map(ctx, mp, "f64")
        s["map"].set_fft(case["fft"])
        s["profile"] = mlc.profile("gaussian", 1.18 * 10.0, 1.0, ref_compat=False)
    elif kind == "expanding":
        s["map"] = mlc.Map(ctx, _map(case["n"], seed, torch.float64), "f64")
        s["loc"] = _locations(case, seed)
        s["base"] = mlc.profile("gaussian", 0.0, WIDTH / case["n"])
    elif kind == "many":
        dt = torch.float64 if case["prec"] == "f64" else torch.float32
        s["map"] = mlc.Map(ctx, _map(case["n"], seed, dt), case["prec"])
        s["map"].set_fft(case["fft"])
        s["profiles"] = [mlc.profile("limb_darkened", r / math.sqrt(2.0), 1.0, ref_compat=False, u=u)
                         for r, u in _limb_profiles(case["nprof"], case["rmax"])]
    elif kind == "ratio":
        s["lc"] = _ratio_inputs(case, seed)
        s["edges"] = mlc.bin_edges(case["nbins"], 1e-4, 300.0, True)
        d, t, sg = (np.array(a) for a in RATIO_DATA)
        s["vars"] = mlc.setup_chi2_calculation((0.4, 0.5), (1.0,), math.sqrt(1750.0 * 850.0 / 1570.0), d, t, sg,
                                               np.array(RATIO_SIZES))
    elif kind == "magdiff":
        s["A"], s["B"], s["w"] = _magdiff_inputs(case, seed)
    elif kind == "fit":
        m = mlc.Map(ctx, _map(case["n"], seed, torch.float32), "f32")
        s["stack"] = mlc.radius_stack(ctx, m, FIT_RADII)
        torch.cuda.synchronize()
        m.close()
        theta, s["off"], s["t"], s["obs"], s["w"] = _fit_inputs(case, seed)
        s["theta"] = theta.requires_grad_(True)
    else:
        s["flux"] = _flux_inputs(case, seed)
    return s


# ----------------------------------------------------------------------------- the calls

def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "step":
        return mlc.convolve_sample_tracks(ctx, s["map"], s["profiles"], s["tracks"], mag=True, pixels=s["pixels"],
                                          out=s["out"])
    if kind == "target":
        s["map"].refresh()
        conv = mlc.convolve(ctx, s["map"], s["profile"])
        chi2, dm = mlc.track_chi2_offset(ctx, conv, 1, *s["tracks"], s["t"], s["obs"], s["w"])
        order = torch.arange(case["ntracks"], dtype=torch.int32, device=DEV)
        best = chi2[0].clone()
        mlc.sort_f64_u32(ctx, best, order)
        hist = mlc.histogram_f64(ctx, best, 100, 0.0, 7.0, log=True)
        return dict(conv=conv, chi2=chi2, dm=dm, best=best, order=order, hist=hist)
    if kind == "expanding":
        s["map"].refresh()
        lc, dlc = mlc.expanding_source(ctx, s["map"], RATIO_SIZES[:case["nsizes"]], s["base"], WIDTH, *s["loc"])
        return dict(lc=lc, dlc=dlc)
    if kind == "many":
        s["map"].refresh()
        if case["nprof"] == 1:
            return mlc.convolve(ctx, s["map"], s["profiles"][0])
        return mlc.convolve_many(ctx, s["map"], s["profiles"])
    if kind == "ratio":
        lca, dlca, lcb, dlcb = s["lc"]
        if case["fused"]:
            bc, be, nper = mlc.pair_bin_fused(ctx, s["vars"], lca, dlca, lcb, dlcb, s["edges"])
            return dict(chi2=bc, exp=be, nper=nper)
        rank, lower, nper = mlc.setup_integral(ctx, lca, lcb, s["edges"])
        chi2 = mlc.calculate_chi2(ctx, s["vars"], lca, dlca, lcb, dlcb, rank)
        bc, be = mlc.bin_chi2(ctx, lower, nper, chi2)
        return dict(rank=rank, lower=lower, nper=nper, pairs=chi2, chi2=bc, exp=be)
    if kind == "magdiff":
        r = mlc.pair_chi2_magdiff(ctx, s["A"], s["B"], s["w"], None, True, nbins=1000, lo=-1.0, hi=9.0, k=case["k"],
                                  want_matrix=case["matrix"])
        return dict(hist=r["hist"], best=r["topk_val"], i=r["topk_i"], j=r["topk_j"])
    if kind == "fit":
        chi2 = mlc.track_chi2(ctx, s["stack"], FIT_RADII, s["theta"], s["off"], s["t"], s["obs"], s["w"])
        (grad,) = torch.autograd.grad(chi2.sum(), s["theta"])
        return dict(chi2=chi2.detach(), grad=grad)
    like, chi2 = mlc.flux_ratio_chi2(ctx, *s["flux"], want_chi2=True)
    return dict(likelihood=like, chi2=chi2)


# ----------------------------------------------------------------------------- what it takes

def _fft_flops(n, maps):
    return maps * 2.5 * n * n * math.log2(float(n) * n)


def work(case):
    """Bytes of every input read once and every output written once, and the arithmetic of the
    transforms, samples and pair sums in operations on numbers of the call's own type."""
    kind = case["kind"]
    n = case.get("n", 0)
    if kind == "step":
        e = 8 if case["prec"] == "f64" else 4
        E = 110.0 * case["ntracks"]
        return dict(bytes=e * (n * n + E * (1 + case["nprof"]) + 4 * case["ntracks"]) + 8 * case["ntracks"],
                    flops=_fft_flops(n, 1 + case["nprof"]) + E * (20 + 12 * case["nprof"]))
    if kind == "target":
        return dict(bytes=8.0 * (2 * n * n + 10 * case["ntracks"]),
                    flops=_fft_flops(n, 2) + 40.0 * case["ntracks"] * case["epochs"])
    if kind == "expanding":
        return dict(bytes=8.0 * (n * n + 2 * case["nsizes"] * case["nloc"]), flops=_fft_flops(n, case["nsizes"]))
    if kind == "many":
        e = 8 if case["prec"] == "f64" else 4
        return dict(bytes=e * float(n) * n * (1 + case["nprof"]), flops=_fft_flops(n, 1 + case["nprof"]))
    if kind == "ratio":
        p = float(case["nloc"]) ** 2
        if case["fused"]:
            return dict(bytes=8.0 * 18 * case["nloc"], flops=p * 40)
        return dict(bytes=p * 12 + 8.0 * 18 * case["nloc"], flops=p * 40)
    if kind == "magdiff":
        return dict(bytes=4.0 * (case["na"] + case["nb"]) * case["epochs"],
                    flops=2.0 * case["na"] * case["nb"] * case["epochs"])
    if kind == "fit":
        E = float(case["ntracks"]) * case["epochs"]
        return dict(bytes=E * (4 * 32 + 12) + case["ntracks"] * 76.0, flops=E * 250)
    N, K = float(case["nloc"]), case["filters"] * case["epochs"]
    return dict(bytes=4.0 * (N * N + 2 * N * K), flops=3.0 * N * N * K)


# ----------------------------------------------------------------------------- 64-bit restatement

def _even(n):
    return n + n % 2


def _raster(shape, rhalf, pix=1.0, u=0.0, compat=False):
    """A profile's normalised raster.  compat: the parameters through six printed decimals and
    a 32-bit float, as the reference passes them."""
    if compat:
        rhalf, pix = (float(np.float32("%f" % x)) for x in (rhalf, pix))
    if shape in ("uniform", "limb_darkened"):
        R = math.sqrt(2.0) * rhalf
        N = _even(2 * (3 + math.ceil(R / pix)))
    elif shape == "gaussian":
        sdev = rhalf / 1.18
        N = _even(math.ceil(4.0 * (1.18 * sdev) / pix))
    else:
        sigma = 0.4106 * rhalf
        N = _even(math.ceil(4.0 * (sigma / 0.4106) / pix))
    c = (np.arange(N) - N // 2) * pix + pix / 2.0
    r = np.hypot(c[None, :], c[:, None])
    if shape == "uniform":
        v = (r < R).astype(np.float64)
    elif shape == "limb_darkened":
        v = np.where(r < R, 1.0 - u * (1.0 - np.sqrt(np.maximum(1.0 - (r / R) ** 2, 0.0))), 0.0)
    elif shape == "gaussian":
        v = np.exp(-r * r / (2 * sdev ** 2))
    else:
        core = 10.0 / (math.exp((rhalf / sigma) ** 0.75) - 1.0)
        edge = sigma * math.log(1.0 + 1.0 / core) ** (4.0 / 3.0)
        v = np.where(r < 2 * rhalf, 1.0 / np.expm1((r / sigma) ** 0.75), 0.0)
        v = np.where(r < edge, core, v)
    return v / v.sum()


def _spectrum(prof, n):
    """Spectrum of a raster wrapped about the origin of an n x n array."""
    N = prof.shape[0]
    k = torch.zeros((n, n), dtype=torch.float64, device=DEV)
    at = (torch.arange(N, device=DEV) - N // 2) % n
    k[at[:, None], at[None, :]] = torch.as_tensor(prof, device=DEV)
    return torch.fft.rfft2(k)


def _convolve(F, prof, n):
    return torch.fft.irfft2(F * _spectrum(prof, n), s=(n, n))


def _cell(x, n):
    """Left pixel and weight of a coordinate on pixel centres j + 1/2 (inside their hull)."""
    j = torch.clamp(torch.floor(x - 0.5), 0, n - 2)
    return j.long(), x - 0.5 - j


def _bilinear(m, x, y):
    n = m.shape[0]
    j, a = _cell(x, n)
    i, d = _cell(y, n)
    f = m.reshape(-1)
    p = i * n + j
    return ((1 - a) * (1 - d) * f[p] + a * (1 - d) * f[p + 1] + (1 - a) * d * f[p + n] + a * d * f[p + n + 1])


def _exact_step(case, seed):
    n = case["n"]
    dt = torch.float64 if case["prec"] == "f64" else torch.float32
    F = torch.fft.rfft2(_map(n, seed, dt).double())
    tr = {k: (a if k == "off" else a.double()) for k, a in _tracks(n, case["ntracks"], seed, dt).items()}
    E = tr["t"].numel()
    out = torch.empty((case["nprof"], E), dtype=torch.float64, device="cpu" if case["host"] else DEV)
    tid = torch.repeat_interleave(torch.arange(case["ntracks"], device=DEV), tr["off"][1:] - tr["off"][:-1])
    c, s = torch.cos(tr["phi"]) * tr["v"], torch.sin(tr["phi"]) * tr["v"]
    for q, (sh, r) in enumerate(_step_profiles(case["nprof"], n)):
        m = _convolve(F, _raster(sh, r), n)
        for e in range(0, E, 20_000_000):
            k, t = tid[e:e + 20_000_000], tr["t"][e:e + 20_000_000]
            z = _bilinear(m, tr["x0"][k] + t * c[k], tr["y0"][k] + t * s[k])
            out[q, e:e + 20_000_000] = -2.5 * torch.log10(z)
    return out


def _exact_target(case, seed):
    n = case["n"]
    mp, (x0, y0, phi, v), t, obs, w = _target_inputs(case, seed)
    conv = _convolve(torch.fft.rfft2(mp), _raster("gaussian", 1.18 * 10.0), n)
    x = x0[:, None] + (v * torch.cos(phi))[:, None] * t
    y = y0[:, None] + (v * torch.sin(phi))[:, None] * t
    r = obs + 2.5 * torch.log10(_bilinear(conv, x, y))
    dm = (w * r).sum(1) / w.sum()
    chi2 = (w * (r - dm[:, None]) ** 2).sum(1)
    return dict(conv=conv, chi2=chi2[None], dm=dm[None], best=torch.sort(chi2)[0], order=None, hist=None)


def _exact_expanding(case, seed):
    n, sizes = case["n"], RATIO_SIZES[:case["nsizes"]]
    mp = _map(n, seed, torch.float64)
    x, y = (torch.as_tensor(a.astype(np.int64), device=DEV) for a in _locations(case, seed))
    F = torch.fft.rfft2(mp)
    cols = [mp[y, x]]
    pix = WIDTH / n
    for z in sizes[1:]:
        cols.append(_convolve(F, _raster("gaussian", z * pix * n / WIDTH, pix, compat=True), n)[y, x])
    lc = torch.stack(cols, 1)
    return dict(lc=lc, dlc=lc[:, 1:] - lc[:, :-1])


def _exact_many(case, seed):
    n = case["n"]
    dt = torch.float64 if case["prec"] == "f64" else torch.float32
    F = torch.fft.rfft2(_map(n, seed, dt).double())
    out = torch.stack([_convolve(F, _raster("limb_darkened", r / math.sqrt(2.0), u=u), n)
                       for r, u in _limb_profiles(case["nprof"], case["rmax"])])
    return out[0] if case["nprof"] == 1 else out


def _exact_ratio(case, seed):
    lca, dlca, lcb, dlcb = _ratio_inputs(case, seed)
    d, t, sg = RATIO_DATA
    sizes, nb = RATIO_SIZES, case["nbins"]
    # the interpolation of every data point on the two images' light curves
    rfac = 23.92865 * math.sqrt(1750.0 * 850.0 / 1570.0)
    chi2 = torch.zeros((case["nloc"], case["nloc"]), dtype=torch.float64, device=DEV)
    inside = []
    for i in range(len(d)):
        m = []
        for mass, lc, dlc in ((0.4, lca, dlca), (0.5, lcb, dlcb)):
            x = t[i] * (1.0 * 8.64 / (rfac * math.sqrt(mass)))
            k = next((k for k in range(len(sizes) - 1) if sizes[k] <= x < sizes[k + 1]), -1)
            m.append(None if k < 0 else lc[:, k] + (x - sizes[k]) / (sizes[k + 1] - sizes[k]) * dlc[:, k])
        inside.append(m[0] is not None or m[1] is not None)
        if not inside[-1]:
            break
        one = torch.ones(case["nloc"], dtype=torch.float64, device=DEV)
        a, b = (one if v is None else v for v in m)
        chi2 += ((d[i] - a[:, None] / b[None, :]) / sg[i]) ** 2
    lo, hi = math.log10(1e-4), math.log10(300.0)
    edges = torch.tensor([10 ** (lo + (i + 1) * (hi - lo) / nb) for i in range(nb)], dtype=torch.float64, device=DEV)
    z, order = torch.sort((lca[:, 0][:, None] / lcb[:, 0][None, :]).reshape(-1), stable=True)
    pairs = chi2.reshape(-1)[order]
    up = torch.searchsorted(z, edges, right=True).tolist()
    bc, be = [], []
    for a, b in zip([0] + up[:-1], up):
        bc.append(pairs[a:b].mean().item() if b > a else 2000.0)
        be.append(torch.exp(-0.5 * pairs[a:b]).mean().item() if b > a else math.exp(-1000.0))
    bc, be = np.array(bc), np.array(be)
    if case["fused"]:
        return dict(chi2=bc, exp=be, nper=None)
    return dict(rank=None, lower=None, nper=None, pairs=pairs, chi2=bc, exp=be)


def _exact_magdiff(case, seed):
    A, B, w = _magdiff_inputs(case, seed)
    k = min(case["k"], case["na"] * case["nb"])
    w = torch.as_tensor(w, device=DEV)

    def side(X):
        X = X.double()
        return (X - (X * w).sum(1, keepdim=True) / w.sum()) * w.sqrt()

    P, Q = side(A), side(B)
    qq = (Q * Q).sum(1)
    # every pair in the expanded form, the smallest ones again as plain sums of squares
    rows = max(1, 200_000_000 // case["nb"])
    thr, val, idx = math.inf, [], []
    for a in range(0, case["na"], rows):
        p = P[a:a + rows]
        c = torch.addmm(qq[None, :] + (p * p).sum(1)[:, None], p, Q.T, alpha=-2.0)
        at = torch.nonzero(c.reshape(-1) < thr).reshape(-1) if math.isfinite(thr) else None
        v = c.reshape(-1) if at is None else c.reshape(-1)[at]
        if v.numel() > k:
            s = torch.topk(v, k, largest=False)
            v, at = s.values, s.indices if at is None else at[s.indices]
        elif at is None:
            at = torch.arange(v.numel(), device=DEV)
        val.append(v)
        idx.append(at + a * case["nb"])
        v, i = torch.cat(val), torch.cat(idx)
        if v.numel() > k:
            s = torch.topk(v, k, largest=False)
            v, i = s.values, i[s.indices]
            thr = v.max().item() * (1 + 1e-9)
        val, idx = [v], [i]
    i = idx[0]
    best = torch.sort(((P[i // case["nb"]] - Q[i % case["nb"]]) ** 2).sum(1))[0]
    return dict(hist=None, best=best.cpu().numpy(), i=None, j=None)


def _fit_rasters(rhalf, N):
    """The smooth thin disc with its flat core on N x N pixels and its derivatives by x, y and
    the half-light radius."""
    c = np.arange(N) - N // 2 + 0.5
    x, y = c[None, :], c[:, None]
    r = np.hypot(x, y)
    sigma = 0.4106 * rhalf
    u = r / sigma
    e = np.exp(u ** 0.75)
    f = 1.0 / (e - 1.0)
    top = 10.0 / (math.exp((rhalf / sigma) ** 0.75) - 1.0)
    outer = f < top
    slope = np.where(outer, -0.75 * u ** -0.25 * e / (e - 1.0) ** 2, 0.0)
    P = np.where(outer, f, top)
    S = P.sum()
    dR = -slope * u / rhalf
    return P / S, slope * x / (r * sigma) / S, slope * y / (r * sigma) / S, dR / S - P / S * dR.sum() / S


def _exact_fit(case, seed):
    n, K = case["n"], len(FIT_RADII)
    N = int(np.ceil(4.4 * FIT_RADII[-1])) // 2 * 2 + 2
    F = torch.fft.rfft2(_map(n, seed, torch.float32).double())
    theta, off, t, obs, w = _fit_inputs(case, seed)
    th = theta.double()
    T = case["epochs"]
    t, obs, w = (a.double().reshape(-1, T) for a in (t, obs, w))
    x0, y0, phi, v, R, dm = (th[:, i:i + 1] for i in range(6))
    vt = v * t
    cs, sn = torch.cos(phi), torch.sin(phi)
    x, y = x0 + vt * cs, y0 + vt * sn
    j, a = _cell(x, n)
    i, d = _cell(y, n)
    nodes = torch.tensor(FIT_RADII, dtype=torch.float64, device=DEV)
    kr = torch.clamp(torch.searchsorted(nodes, R.contiguous(), right=True) - 1, 0, K - 2)
    h = nodes[kr + 1] - nodes[kr]
    s = (R - nodes[kr]) / h

    def herm(s):
        return ((2 * s ** 3 - 3 * s ** 2 + 1, 3 * s ** 2 - 2 * s ** 3), (s ** 3 - 2 * s ** 2 + s, s ** 3 - s ** 2),
                (6 * s * s - 6 * s, 6 * s - 6 * s * s), (3 * s * s - 4 * s + 1, 3 * s * s - 2 * s))

    (rv, rt, rdv, rdt), (xv, xt, xdv, xdt), (yv, yt, ydv, ydt) = herm(s), herm(a), herm(d)
    M = Mx = My = MR = 0.0
    for k in range(K):
        fields = [_convolve(F, p, n).reshape(-1) for p in _fit_rasters(FIT_RADII[k], N)]
        for side in (0, 1):  # this radius as the lower and as the upper end of a track's bracket
            rows = torch.nonzero((kr[:, 0] + side) == k).reshape(-1)
            if rows.numel() == 0:
                continue
            z = [torch.zeros((case["ntracks"], T), dtype=torch.float64, device=DEV) for _ in range(4)]
            sub = lambda q: q[rows]  # noqa: E731
            wv, wt, wdv, wdt = sub(rv[side]), sub(rt[side]) * sub(h), sub(rdv[side]) / sub(h), sub(rdt[side])
            for ay in (0, 1):
                for ax in (0, 1):
                    p = (sub(i) + ay) * n + sub(j) + ax
                    m, fx, fy, fr = (f[p] for f in fields)
                    Mc, McR = wv * m + wt * fr, wdv * m + wdt * fr
                    Xc, XcR, Yc, YcR = wv * fx, wdv * fx, wv * fy, wdv * fy
                    vx, tx, dvx, dtx = (sub(q[ax]) for q in (xv, xt, xdv, xdt))
                    vy, ty, dvy, dty = (sub(q[ay]) for q in (yv, yt, ydv, ydt))
                    z[0][rows] += vx * vy * Mc + tx * vy * Xc + vx * ty * Yc
                    z[1][rows] += dvx * vy * Mc + dtx * vy * Xc + dvx * ty * Yc
                    z[2][rows] += vx * dvy * Mc + tx * dvy * Xc + vx * dty * Yc
                    z[3][rows] += vx * vy * McR + tx * vy * XcR + vx * ty * YcR
            M, Mx, My, MR = M + z[0], Mx + z[1], My + z[2], MR + z[3]
    r = obs - (-2.5 * torch.log10(M) + dm)
    gm = -2 * w * r
    gq = gm * -2.5 / (math.log(10.0) * M)
    gx, gy = gq * Mx, gq * My
    grad = torch.stack([gx.sum(1), gy.sum(1), (vt * (cs * gy - sn * gx)).sum(1), (t * (cs * gx + sn * gy)).sum(1),
                        (gq * MR).sum(1), gm.sum(1)], 1)
    return dict(chi2=(w * r * r).sum(1), grad=grad)


def _exact_flux(case, seed):
    fo, dfo, m1, m2 = _flux_inputs(case, seed)
    N, K = case["nloc"], case["filters"] * case["epochs"]
    fo, dfo = (torch.as_tensor(a.astype(np.float64).reshape(-1), device=DEV) for a in (fo, dfo))
    m1, m2 = m1.reshape(N, K).double(), m2.reshape(N, K).double()
    chi2 = torch.zeros((N, N), dtype=torch.float64, device=DEV)
    for k in range(K):
        chi2 += 0.5 * ((fo[k] - m1[:, k][None, :] / m2[:, k][:, None]) / dfo[k]) ** 2
    return dict(likelihood=torch.exp(-chi2).sum().item(), chi2=chi2)


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)
