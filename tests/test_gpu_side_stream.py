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
