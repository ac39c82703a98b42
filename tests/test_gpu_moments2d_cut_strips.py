"""Strips that the support cuts beside crowded ones: the targets' windows there may
cover each other or lie far apart, in one strip or in several."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

REL = 1e-5  # the repository's bar per density
H = 0.75


@pytest.fixture
def mctx():
    from entropical_gb300 import Context
    c = Context(0)
    c.set_tuning(pair_variant=[None, 7, None], moment_cells_per_h=3)
    yield c
    c.close()


def points(n, span, sparse, strips, cut, offset=0.0):
    """A few targets on the lowest edge of `strips` strips, and n points in those two
    strips above, on both sides of the targets' support in y (cut) or inside it."""
    rng = np.random.default_rng(n)
    w = H / 3 * (1 + 1e-4)  # the width of a strip
    low = [q * (w + 1e-6) for q in range(strips)]
    ys = np.repeat(low, sparse // strips)
    xs = np.tile(np.linspace(-span, span, sparse // strips), strips)
    q = np.arange(n) % strips
    top = H + (3e-5 if cut else -1e-3)
    yc = np.array(low)[q] + np.where(rng.random(n) < 0.5, 0.6, top)
    x = np.append(xs, rng.uniform(-span, span, n)) + offset
    return np.stack([x, np.append(ys, yc)]).astype(np.float32), len(xs)


@pytest.mark.parametrize("strips", [1, 2])
@pytest.mark.parametrize("sparse", [2, 32, 96, 2000])
@pytest.mark.parametrize("n,span", [(500, 200.0), (20_000, 200.0), (20_000, 6.0), (20_000, 1.2)])
def test_sums_of_cut_strips(mctx, n, span, sparse, strips):
    for offset in (0.0, 5000.0):  # 96-byte and 128-byte rows
        x, m = points(n, span, sparse, strips, True, offset)
        p = mctx.combined_densities(x, None, [0, 1], [H, H])
        t = np.unique(np.append(np.arange(m), np.linspace(0, x.shape[1] - 1, 50))).astype(np.uint32)
        ref = O.density_fp64(x, [H, H], targets=t)
        assert np.max(np.abs(p[t] - ref) / ref) < REL


@pytest.mark.parametrize("strips", [1, 2])
def test_windows_apart_do_not_hold_the_kernel_up(mctx, strips):
    # 32 targets with windows of some 2,000 of 600,000 sources: what they add to the
    # target kernel is a few times the kernel without them, not the whole union of
    # their windows (a hundred times it)
    ms = {}
    for cut in (False, True):
        x, _ = points(600_000, 200.0, 32, strips, cut)
        t = []
        for _ in range(5):
            mctx.entropy_batch([(x, [H, H])])
            t.append(mctx.last_stats().moment_target_ms)
        ms[cut] = min(t)
    assert ms[True] < 10 * ms[False], ms
