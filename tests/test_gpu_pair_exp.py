"""The exponentials of the ratio statistic are as exact as the library's: bins of one pair hold the
bare exp(-chi2/2)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def test_bin_of_one_pair_is_the_rounded_exponential(ctx):
    import microsn_gb300 as mlc
    n = 200_000
    rng = np.random.default_rng(4)
    c = np.concatenate([rng.uniform(0, 1400, n // 2), np.exp(rng.uniform(-40, np.log(1400.0), n // 2 - 8)),
                        [0.0, 1e-300, 1.0, 1399.999, 1400.0, 1480.0, 1600.0, np.inf]])
    chi2 = torch.as_tensor(c, device=DEV)
    lower = np.arange(n, dtype=np.uint32)
    bc, be = mlc.bin_chi2(ctx, lower, np.ones(n, np.uint32), chi2)
    assert np.array_equal(bc, c)
    want = np.exp(-c.astype(np.longdouble) / 2)
    normal = want >= 2.3e-308
    err = np.abs(be[normal].astype(np.longdouble) / want[normal] - 1)
    # correctly rounded up to 0.03 ulp: 2^-53 at most, and the remainder of the series (2^-57)
    assert float(err.max()) <= 2.0 ** -53 * 1.07
    assert np.all(np.abs(be[~normal] - want[~normal].astype(np.float64)) <= 5e-324)
