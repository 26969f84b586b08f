"""The tensor-core pair kernel's epilogue (csrc/pairtc.cu) at the edges of its 128 x 48 tiles, for
each of its widths: single near-identical pairs send one lane of a warp through the exact
path, the others are counted in the packed one."""
import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("epi", [12, 16, 24])
@pytest.mark.parametrize("NA,NB,T", [(128, 48, 128), (129, 97, 65), (257, 49, 64), (1, 1, 3), (640, 480, 128)])
def test_histogram_and_topk_at_tile_edges(epi, NA, NB, T):
    import microsn_gb300 as mlc
    ctx = mlc.Context()
    K = 64 if T <= 64 else 128
    for lg in range(12):
        ctx.tune_set(f"pairdiff_tc K{K} bins1024 pairs~4^{lg}", epi)
    rng = np.random.default_rng(NA + NB + T)
    A = np.cumsum(rng.normal(0, 0.05, (NA, T)), axis=1).astype(np.float32)
    B = np.cumsum(rng.normal(0, 0.05, (NB, T)), axis=1).astype(np.float32)
    for c in range(0, min(NB, NA), 11):
        B[c] = A[(7 * c) % NA] + rng.normal(0, 1e-4, T).astype(np.float32)
    w = 1.0 / rng.uniform(0.02, 0.1, T) ** 2
    k = min(20, NA * NB)
    # the range's ends lie inside the values: counts below and above it
    r = mlc.pair_chi2_magdiff(ctx, torch.as_tensor(A, device="cuda"), torch.as_tensor(B, device="cuda"), w, None, False,
                              method="tensor", nbins=200, lo=-1, hi=3.5, k=k)
    ref = oracle.pair_chi2_magdiff(A, B, w, np.zeros(T), False)
    # FP32 assembly within 4e-6 of chi2, and the bin's arithmetic (lg2 within 2^-22, t below 2^9)
    counts, near = oracle.histogram(ref, 200, -1, 3.5, log=True, rel_tol=1e-5)
    assert np.abs(r["hist"].astype(np.int64) - counts.astype(np.int64)).sum() <= 2 * near
    st = r["stats"]
    assert int(r["hist"].sum()) + st["below"] + st["above"] == NA * NB
    assert abs(st["below"] - int((ref < 0.1).sum())) <= near
    np.testing.assert_allclose(r["topk_val"], np.sort(ref)[:k], rtol=1e-6)
    ctx.close()
