"""The terms of the reference's mutual-information formula, p_ij log(p_ij / p_i / p_j)
in the float log, at bandwidths across the float range: the densities reach 1e60 and
1e-60, their products 1e120 and 1e-120. Against the formula over the densities of
single calls (joint densities are FP32 sums, within 1e-6 of each other)."""
import numpy as np
import pytest

from entropical_gb300.densities import REF_MI

pytestmark = pytest.mark.gpu

LOG_ULPS = 2 * 2.0 ** -23  # of the float log
ARG = 2.0 ** -23  # the log's argument, rounded to float
DENSITY = 1e-6


@pytest.mark.parametrize("hs", [(0.3, 0.2, 0.5), (1e-30, 1e-30, 1e-30), (1e30, 1e30, 1e30),
                                (1e-30, 0.3, 1e30), (1e-37, 1e-37, 1e-3)])
@pytest.mark.parametrize("n", [1, 777, 3000])
def test_terms(ctx, n, hs):
    rng = np.random.default_rng(n)
    x = rng.standard_normal((3, n)).astype(np.float32)
    x[:, n // 2:] = np.round(x[:, n // 2:] * 4) / 4  # ties, so that tiny supports hold pairs
    h = list(hs)
    p = [ctx.combined_densities(x, None, [i], [h[i]], compat_norm=True) for i in range(3)]
    got = ctx.reference_estimator(x, h, REF_MI)
    for i in range(3):
        for j in range(i + 1, 3):
            pij = ctx.combined_densities(x, None, [i, j], [h[i], h[j]], compat_norm=True)
            log = np.log(pij / p[i] / p[j])
            tol = (pij * (LOG_ULPS * np.abs(log) + ARG + DENSITY * (np.abs(log) + 1))).sum()
            assert np.isfinite(got[i, j])
            assert abs(got[i, j] - (pij * log).sum()) <= tol
            assert got[j, i] == got[i, j]
