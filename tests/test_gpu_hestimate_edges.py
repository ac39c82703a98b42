"""The bandwidth search's kernels at the edges of their tiles: 256 values per
chunk of the rule of thumb, 128 targets per warp and 1,024 per block of the
convolution, 2,048 values per prefix chunk; columns whose values need a far
shifted fixed point, and sorts without an order."""
import numpy as np
import pytest

from entropical_gb300 import workloads
from entropical_gb300.densities import HEST_AMISE, HEST_THUMB
from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [2, 127, 128, 129, 255, 256, 257, 1023, 1024, 1025, 2047, 2048, 2049, 6147]
# three float roundings of the value: the sum, n^2 and their quotient
TOL = 3 * 2.0 ** -24


@pytest.mark.parametrize("n", SIZES)
def test_convolution_at_tile_edges(ctx, n):
    x = np.sort(workloads.gmm_1d(n, seed=n))
    for h in (1e-4, 0.05, 2.0):
        ref = O.epa_conv_fp64(x, h)
        assert abs(ctx.epa_convolution(x, h) - ref) <= TOL * ref


@pytest.mark.parametrize("scale,offset", [(1e-30, 0.0), (1e25, 0.0), (1.0, 3e4), (2e-3, -70.0)])
def test_convolution_far_scales_and_offsets(ctx, scale, offset):
    x = np.sort((workloads.gmm_1d(3001, seed=8).astype(np.float64) * scale + offset)
                .astype(np.float32))
    for h in (0.01 * scale, 0.3 * scale):
        ref = O.epa_conv_fp64(x, h)
        assert abs(ctx.epa_convolution(x, h) - ref) <= TOL * ref


@pytest.mark.parametrize("n", SIZES)
def test_search_at_tile_edges(ctx, n):
    rng = np.random.default_rng(n)
    cols = np.stack([workloads.mixture_instance(rng, 1, n)[0] for _ in range(3)])
    t, _ = ctx.hestimate(cols, HEST_THUMB)
    h, st = ctx.hestimate(cols, HEST_AMISE)
    for c, tc, hc in zip(cols, t, h):
        assert tc == np.float32(O.thumb_ref(c))
        assert hc == np.float32(O.hestimate_amise(c, exact=False)[0])


def test_constant_column(ctx):
    x = np.stack([np.full(500, 0.25, np.float32), workloads.gmm_1d(500, seed=3)])
    h, _ = ctx.hestimate(x, HEST_AMISE)
    assert h[0] == 0.0 and h[1] > 0.0  # no spread: the bracket [0, 0]
    assert abs(ctx.epa_convolution(x[0], 0.1) - 4.5) <= TOL * 4.5
