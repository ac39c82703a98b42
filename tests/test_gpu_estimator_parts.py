"""The estimators' sums in parts: one part up to 1,024 values, then one more per
1,024 values while the GPU has room; many columns take one part each. Against
the formulas over the densities of single calls (1-D densities are exact, so
only the float logarithm differs, by 2 units in its last place at most)."""
import numpy as np
import pytest

from entropical_gb300.densities import REF_KLDIV, REF_NEGS

pytestmark = pytest.mark.gpu

LOG_ULPS = 2 * 2.0 ** -23


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 3000, 16 * 1024 + 7])
@pytest.mark.parametrize("m", [2, 3])
def test_parts(ctx, n, m):
    rng = np.random.default_rng(n + m)
    x = rng.standard_normal((m, n)).astype(np.float32)
    h = [0.3] * m
    p = [ctx.combined_densities(x, None, [i], [h[i]], compat_norm=True) for i in range(m)]
    q = [v / v.sum() for v in p]
    got = ctx.reference_estimator(x, h, REF_NEGS)
    for i in range(m):
        t = q[i] * np.log(q[i])
        assert abs(got[i] + t.sum()) <= LOG_ULPS * np.abs(t).sum() + 1e-12
    kl = ctx.reference_estimator(x, h, REF_KLDIV)
    for i in range(m):
        for j in range(m):
            if i == j:
                assert kl[i, j] == 0.0
                continue
            t = q[i] * np.log(q[i] / q[j])
            # the logarithm's float argument is rounded as well
            assert abs(kl[i, j] - t.sum()) <= LOG_ULPS * (np.abs(t).sum() + 1.0)
    d = ctx.dens_all(x, h, 1)
    assert np.allclose(d, np.array(q), rtol=1e-12, atol=0)


def test_many_columns_take_one_part(ctx):
    rng = np.random.default_rng(3)
    x = rng.standard_normal((1300, 1500)).astype(np.float32)
    h = [0.3] * len(x)
    got = ctx.reference_estimator(x, h, REF_NEGS)
    few = ctx.reference_estimator(x[:2], h[:2], REF_NEGS)
    assert np.allclose(got[:2], few, rtol=1e-13, atol=0)  # the order of the FP64 sums
