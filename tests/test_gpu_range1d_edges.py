"""The 1-D range sums at the edges of their shapes: 32 targets per warp, 256 per
block, 2,048 points per step of the one-kernel prefix (up to 4,096 points) and
per chunk of the three-kernel one; log-sums and densities from the kernel's own
epilogue."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 255, 256, 257, 511, 512, 513, 2047, 2048, 2049, 4095, 4096, 4097, 9001]
REL = 1e-5  # the repository's bar per density


def _column(n):
    rng = np.random.default_rng(n)
    x = rng.standard_normal(n).astype(np.float32)
    x[: n // 3] = np.round(x[: n // 3], 1)  # ties
    if n > 40:
        x[7] = 50.0  # alone in its support
    return x


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("h", [1e-3, 0.2, 1e3])
def test_densities(ctx, n, h):
    x = _column(n)
    p = ctx.combined_densities(x, n, [0], [h])
    ref = O.density_fp64(x[None], [h])
    assert np.max(np.abs(p - ref) / ref) < REL


@pytest.mark.parametrize("h", [0.05, 2.0])
def test_entropies_short_and_long_in_batches(ctx, h):
    # a batch of short instances (one prefix kernel) and one with a longer one
    short = [(_column(n), [h]) for n in SIZES if n <= 4096]
    H = ctx.entropy_batch(short)
    mixed = ctx.entropy_batch(short + [(_column(9001), [h])])
    # the sums are exact, their logs exact integers: the same bits
    assert np.array_equal(H, mixed[:-1])
    for (x, hh), v in zip(short, H):
        assert abs(v - O.entropy_fp64(x[None], hh)) < 1e-6
