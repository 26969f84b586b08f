"""Calls on a stream that does not wait for the legacy default stream (torch's side streams) and
is still busy: their tables and results go through that stream, so that a call neither
overwrites what the one before it still reads nor reads what is not there yet."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture
def side():
    """A context on a side stream, and a function that keeps the stream busy for some 10 ms."""
    import microsn_gb300 as mlc
    s = torch.cuda.Stream()
    c = mlc.Context(0, stream=s)
    torch.cuda.synchronize()
    yield c, s, lambda: torch.cuda._sleep(20_000_000)
    torch.cuda.synchronize()
    c.close()


def _vars(d, s):
    import microsn_gb300 as mlc
    return mlc.Chi2Vars(3, np.array([0, 1, -1], np.int32), np.array([1, -1, 0], np.int32), np.array([0.3, 0.6, 0.0]),
                        np.array([0.2, 0.0, 0.9]), np.array(d), np.array(s), 0.0)


def test_ratio_chi2_of_two_calls_in_a_row(ctx, side):
    import microsn_gb300 as mlc
    c, s, busy = side
    rng = np.random.default_rng(3)
    A, B = (torch.as_tensor(np.exp(rng.normal(0, 0.5, (300, 3))), device=DEV) for _ in range(2))
    dA, dB = torch.diff(A, dim=1).contiguous(), torch.diff(B, dim=1).contiguous()
    both = [_vars([0.7, 1.2, 1.1], [0.1, 0.15, 0.3]), _vars([1.7, 0.4, 0.9], [0.2, 0.05, 0.6])]
    want = [mlc.calculate_chi2(ctx, v, A, dA, B, dB).clone() for v in both]
    edges = mlc.bin_edges(50, 1e-2, 1e2)
    fused = [mlc.pair_bin_fused(ctx, v, A, dA, B, dB, edges) for v in both]
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        mlc.calculate_chi2(c, both[0], A, dA, B, dB)  # (workspaces made)
        s.synchronize()
        busy()
        got = [mlc.calculate_chi2(c, v, A, dA, B, dB) for v in both]
        busy()
        binned = [mlc.pair_bin_fused(c, v, A, dA, B, dB, edges) for v in both]
    s.synchronize()
    for w, g in zip(want, got):
        assert torch.equal(w, g)
    for w, g in zip(fused, binned):
        assert np.array_equal(w[2], g[2])
        for k in range(2):
            np.testing.assert_allclose(g[k], w[k], rtol=1e-13)  # (sums of 90000 values in no fixed order)


def test_convolution_of_two_profiles_in_a_row(ctx, side):
    import microsn_gb300 as mlc
    c, s, busy = side
    mp = torch.rand((360, 360), dtype=torch.float64, device=DEV)
    profs = [mlc.profile("gaussian", 3.0, 1.0, ref_compat=False), mlc.profile("gaussian", 4.0, 1.0, ref_compat=False)]
    m = mlc.Map(ctx, mp, "f64")
    want = [mlc.convolve(ctx, m, p).clone() for p in profs]
    m.close()
    with torch.cuda.stream(s):
        m = mlc.Map(c, mp, "f64")
        busy()
        got = [mlc.convolve(c, m, p) for p in profs]
        s.synchronize()
        m.close()
    for w, g in zip(want, got):
        assert torch.equal(w, g)


@pytest.mark.parametrize("k", [50, 3000])
def test_best_pairs(ctx, side, k):
    import microsn_gb300 as mlc
    c, s, busy = side
    g = torch.Generator(device=DEV).manual_seed(1)
    A, B = (torch.cumsum(torch.randn((n, 40), generator=g, device=DEV) * 0.1, 1).contiguous() for n in (700, 900))
    w = np.full(40, 400.0)
    want = mlc.pair_chi2_magdiff(ctx, A, B, w, None, True, nbins=100, lo=-1.0, hi=9.0, k=k)
    torch.cuda.synchronize()
    for _ in range(3):
        with torch.cuda.stream(s):
            busy()
            got = mlc.pair_chi2_magdiff(c, A, B, w, None, True, nbins=100, lo=-1.0, hi=9.0, k=k)
        for name in ("hist", "topk_val", "topk_i", "topk_j"):
            assert np.array_equal(np.asarray(want[name]), np.asarray(got[name])), name


def test_offset_chi2_of_two_calls_in_a_row(ctx, side):
    import microsn_gb300 as mlc
    c, s, busy = side
    m = torch.rand((500, 30), dtype=torch.float64, device=DEV)
    obs = [np.linspace(0, 1, 30), np.linspace(1, -1, 30)]
    w = [np.full(30, 9.0), np.linspace(1, 4, 30)]
    want = [mlc.chi2_offset(ctx, m, o, x) for o, x in zip(obs, w)]
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        busy()
        got = [mlc.chi2_offset(c, m, o, x) for o, x in zip(obs, w)]
    s.synchronize()
    for a, b in zip(want, got):
        assert all(torch.equal(p, q) for p, q in zip(a, b))
