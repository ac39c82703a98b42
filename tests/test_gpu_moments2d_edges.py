"""The strip-moment kernels at the edges of their shapes: 16 targets per round
and 32 per warp, 128 per block, 2,048 points per prefix chunk, 3 to 23 inside
strips; batches that mix instances near the origin (64-bit coefficients, 96-byte
rows) with instances far from it (128-bit, 128-byte), whose kernels run apart."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

REL = 1e-5  # the repository's bar per density


@pytest.fixture
def mctx():
    from entropical_gb300 import Context
    c = Context(0)
    c.set_tuning(pair_variant=[None, 7, None])
    yield c
    c.close()


@pytest.mark.parametrize("n", [15, 16, 17, 31, 32, 33, 127, 128, 129, 2047, 2048, 2049, 4133])
@pytest.mark.parametrize("cells", [2, 3, 12])
def test_shapes(mctx, n, cells):
    mctx.set_tuning(moment_cells_per_h=cells)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((2, n)).astype(np.float32)
    x[1, : n // 2] = x[1, 0]  # half of the points in one strip
    h = [0.7, 0.4]
    p = mctx.combined_densities(x, None, [0, 1], h)
    ref = O.density_fp64(x, h)
    assert np.max(np.abs(p - ref) / ref) < REL


def test_near_and_far_instances_in_one_batch(mctx):
    rng = np.random.default_rng(5)
    insts = []
    for q, n in enumerate([900, 128, 2500, 33, 1, 4100, 640]):
        x = rng.standard_normal((2, n)).astype(np.float32)
        if q % 2:  # scaled coordinates on either side of 2^8
            x += np.float32([[60.0 if q == 1 else 3e3], [-1e4 if q == 3 else 0.0]])
        insts.append((x, [0.3, 0.25]))
    H = mctx.entropy_batch(insts)
    for (x, h), v in zip(insts, H):
        alone = mctx.entropy_batch([(x, h)])[0]
        # the same exact sums; FP32 edge sums shared out differently
        assert abs(v - alone) < 1e-7
        assert abs(v - O.entropy_fp64(x, h)) < 1e-6


def test_every_point_near_the_bound_of_the_64_bit_form(mctx):
    # scaled coordinates just below and just above 2^8 (h 2^k = 0.625)
    rng = np.random.default_rng(6)
    for top in (255.9, 256.1):
        x = (rng.uniform(-1, 1, (2, 3000)) * 4).astype(np.float32)
        x[:, 0] = np.float32(top)
        x[:, 1] = np.float32(-top)
        p = mctx.combined_densities(x, None, [0, 1], [0.625, 0.625])
        ref = O.density_fp64(x, [0.625, 0.625])
        assert np.max(np.abs(p - ref) / ref) < REL


@pytest.mark.parametrize("n", [40, 333, 6001])
@pytest.mark.parametrize("cells", [2, 3, 12])
def test_inside_strips_that_cross_the_support(mctx, n, cells):
    # y on the lowest edge of the first strip and one bandwidth above it, give or
    # take roundings: inside strips whose sources are partly out of the support,
    # summed pair by pair for one target of a warp or for all of them
    mctx.set_tuning(moment_cells_per_h=cells)
    rng = np.random.default_rng(n)
    h = np.float32(0.75)
    y = np.where(rng.random(n) < 0.5, 0.0, h * (1 + rng.integers(-4, 5, n) * 2.0**-23))
    few = rng.random(n) < 0.2
    y[few] = rng.random(few.sum()) * 2
    y[0] = 0.0
    x = np.stack([rng.standard_normal(n), y]).astype(np.float32)
    p = mctx.combined_densities(x, None, [0, 1], [0.5, h])
    ref = O.density_fp64(x, [0.5, h])
    assert np.max(np.abs(p - ref) / ref) < REL


@pytest.mark.parametrize("n", [256_400, 257_000])
def test_moment_sums_near_the_bounds_of_their_fields(mctx, n):
    # n max|x^2 y| just below and just above 4.3e12 (scaled coordinates, h 2^k =
    # 0.625): 96-byte rows with nearly full fields of either sign, or 128-byte rows
    rng = np.random.default_rng(n)
    sign = rng.choice(np.float32([-1, 1]), (2, n))
    x = (sign * (255.9 - 4 * rng.random((2, n)) ** 4)).astype(np.float32)
    h = [0.625, 0.625]
    p = mctx.combined_densities(x, None, [0, 1], h)
    t = np.linspace(0, n - 1, 64).astype(np.uint32)
    ref = O.density_fp64(x, h, targets=t)
    assert np.max(np.abs(p[t] - ref) / ref) < REL


def test_light_tiles_by_warps_and_by_blocks():
    # 2-D slots of a batch with strip moments run from a work list; with at least
    # 512 slots per SM, light ones by one warp each. The same instances in a
    # smaller batch run by blocks: the same FP32 sums, so the same entropies up
    # to the order of FP64 additions. Instances below the moments' support
    # (several runs per tile, some joined) share the list.
    from entropical_gb300 import Context
    ctx = Context(0)
    rng = np.random.default_rng(17)
    n = 20_000
    a = np.tanh(2 * rng.standard_normal((2, n))).astype(np.float32)  # crowded edge strips
    b = rng.standard_normal((2, n)).astype(np.float32)
    c = (np.round(rng.standard_normal((2, n)) * 400) / 400).astype(np.float32)
    c[:, :500] = c[:, :1]
    kinds = [(a, [0.5, 0.6]), (b, [0.8, 0.8]), (c, [0.03, 0.02]), (c[:, :37], [0.03, 0.02])]

    def batch(copies):
        H = ctx.entropy_batch(kinds * copies).reshape(copies, len(kinds))
        st = ctx.last_stats()
        assert st.moment_edge_ms > 0  # the strip moments ran
        return H, st.tiles

    few, tiles = batch(40)
    assert 2432 < tiles < 512 * 132  # no tile shared out; fewer slots than the rule on any SM count
    many, tiles = batch(170)
    assert tiles > 512 * 160
    assert np.allclose(few, few[0], rtol=1e-12, atol=0)
    assert np.allclose(many, few[0], rtol=1e-12, atol=0)
    ctx.close()
    for q in range(4):
        assert abs(few[0, q] - O.entropy_fp64(*kinds[q])) < 1e-6


def test_heavy_tiles_in_shares():
    # crowded strips: tiles of one to twenty-odd chunks of 1,536 sources, whose
    # chunks go to eight CTAs; the shares add the same FP32 chunk sums
    from entropical_gb300 import Context
    rng = np.random.default_rng(23)
    insts = []
    for n in (6_000, 12_289, 20_000, 33_001):
        x = rng.standard_normal((2, n)).astype(np.float32)
        # most points in two narrow bands a support's edge apart: the tiles of one
        # have the other as their edge strip, with all of it inside the x-window
        x[1, : 2 * n // 3] = np.where(rng.random(2 * n // 3) < 0.5, 0.0, 0.79) \
            + rng.random(2 * n // 3) * 0.02
        insts.append((np.ascontiguousarray(x), [2.5, 0.8]))
    ctx = Context(0)
    ctx.set_tuning(pair_variant=[None, 7, None])
    got = ctx.entropy_batch(insts)
    big = ctx.entropy_batch(insts * 30)  # more slots per SM: other tiles in shares
    for q, (x, h) in enumerate(insts):
        assert abs(got[q] - O.entropy_fp64(x, h)) < 1e-6
        assert np.allclose(big[q::4], got[q], rtol=1e-12, atol=0)
    ctx.close()
