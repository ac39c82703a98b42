"""Convolutions at one bandwidth on columns whose range is large against it: a bulk
on the scale of h beside outliers that the fixed point of the prefix sums must not
be scaled by."""
import numpy as np
import pytest

from entropical_gb300.densities import HEST_AMISE
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# three float roundings of the value: the sum, n^2 and their quotient
TOL = 3 * 2.0 ** -24


def check(ctx, x, h):
    x = np.sort(np.asarray(x).astype(np.float32))
    h = float(np.float32(h))
    ref = O.epa_conv_fp64(x, h)
    assert abs(ctx.epa_convolution(x, h) - ref) <= TOL * ref


@pytest.mark.parametrize("out", [1e6, -1e6, 6.4e7, 1e12, -1e30, 3e38])
@pytest.mark.parametrize("bulk", [1e-10, 1e-7, 1e-4])
@pytest.mark.parametrize("n", [2, 1000, 2049])
def test_bulk_beside_an_outlier(ctx, n, bulk, out):
    rng = np.random.default_rng(n)
    x = np.append(bulk * rng.random(n - 1), out)
    for h in (bulk / 10, bulk, 10 * bulk):
        check(ctx, x, h)


@pytest.mark.parametrize("h", [1e-7, 3e-8, 1.5e-8])
def test_two_values_beside_an_outlier(ctx, h):
    x = np.append(np.where(np.arange(2000) % 2, 0.0, 4e-8), 6.4e7)
    check(ctx, x, h)


def test_outliers_on_both_sides(ctx):
    # pairs of outliers in each other's support, and a bulk with an offset
    rng = np.random.default_rng(5)
    x = np.concatenate([[-1e30, -1e30, 1e20, 1e20, 1e20], 7.0 + 1e-3 * rng.standard_normal(3000)])
    for h in (1e-5, 1e-3, 1.0, 1e22):
        check(ctx, x, h)


def test_bandwidths_at_the_ends_of_the_float_range(ctx):
    rng = np.random.default_rng(6)
    check(ctx, np.append(rng.random(500) * 1e-37, 1.0), 2e-38)  # differences near the smallest normal floats
    check(ctx, rng.standard_normal(500), 3e38)  # 2h overflows a float: every pair counts


@pytest.mark.parametrize("out", [50.0, 1e4, -1e9, 1e15])
def test_search_beside_an_outlier(ctx, out):
    # the search's bandwidths grow with the outlier: its unit may follow the range
    rng = np.random.default_rng(7)
    cols = np.stack([np.append(rng.standard_normal(2048), out),
                     np.append(1e-3 * rng.integers(0, 2, 2048), out)]).astype(np.float32)
    h, _ = ctx.hestimate(cols, HEST_AMISE)
    for c, hc in zip(cols, h):
        assert hc == np.float32(O.hestimate_amise(c, exact=False)[0])
