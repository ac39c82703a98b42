"""The device sort and tile plan at the sizes where their forms change: radix
chunks of 2,048 values, segments of up to two chunks that one block sorts,
segments whose scatter blocks sum their own histogram rows (small sorts) or read
a prefix kernel's, and non-finite input anywhere in a column; batches planned by a group of lanes per slot (up to 131,072 slots)
or by a thread."""
import numpy as np
import pytest

from entropical_gb300 import _native
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CHUNK = 2048


def _ties(rng, n):
    """Values with many ties, both signs and both zeros."""
    x = (np.round(rng.standard_normal(n) * 500) / 500).astype(np.float32)
    x[rng.integers(0, n, max(1, n // 50))] = np.float32(-0.0)
    return x


@pytest.mark.parametrize("n", [1, 31, CHUNK - 1, CHUNK, CHUNK + 1,
                               2 * CHUNK - 1, 2 * CHUNK, 2 * CHUNK + 1, 3 * CHUNK + 5,
                               256 * CHUNK, 256 * CHUNK + 1])
def test_sort_at_chunk_edges(ctx, n):
    # 2 chunks: the largest segment sorted in one block; 256 chunks: the largest
    # column whose scatter blocks sum the rows themselves
    rng = np.random.default_rng(n)
    x = _ties(rng, n)
    lo, hi = ctx.neighbor_windows(x, 0.01)
    lo2, hi2 = O.boxes(x, 0.01)
    assert np.array_equal(lo, lo2) and np.array_equal(hi, hi2)


@pytest.mark.parametrize("n_cols,n", [(1, 5000), (300, 30011)])
def test_many_columns_sort_as_one(ctx, n_cols, n):
    # 300 x 15 chunks: the large form; each column's entropy equals a call of its own
    rng = np.random.default_rng(n_cols)
    cols = [rng.standard_normal(n).astype(np.float32) for _ in range(n_cols)]
    H = ctx.entropy_batch([(c, [0.2]) for c in cols])
    for q in {0, n_cols // 2, n_cols - 1}:
        one = ctx.entropy_batch([(cols[q], [0.2])])[0]
        assert H[q] == one  # exact 1-D sums, the same blocks of log-sums


@pytest.mark.parametrize("at", [0, CHUNK - 1, CHUNK, 9_999])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_anywhere_is_an_error(ctx, at, bad):
    x = np.linspace(-1, 1, 10_000, dtype=np.float32)
    x[at] = bad
    with pytest.raises(_native.NativeError) as e:
        ctx.combined_densities(x, x.size, [0], [0.1])
    assert e.value.status == 5
    x[at] = 0.5
    assert np.all(ctx.combined_densities(x, x.size, [0], [0.1]) > 0)


@pytest.mark.parametrize("d,h,cells3,few,many", [
    (1, 0.3, 1, 200, 6000), (2, 0.3, 1, 100, 2000), (2, 1e-3, 1, 20, 50), (3, 0.3, 1, 100, 230),
    (3, 1e-3, 1, 20, 50), (3, 0.3, 2, 30, 70)])
def test_plan_by_group_and_by_thread(d, h, cells3, few, many):
    # the same density in a batch of at most 131,072 slots, planned by 16 lanes
    # per slot (32 with 25 runs around a tile), and in one of more, planned by
    # threads: the same tiles and runs, so the same sums up to the order of the
    # FP64 additions. Tiny h: thousands of strips of a few points, runs joined
    # across strips.
    from entropical_gb300 import Context
    rng = np.random.default_rng(7 * d)
    n = 3001
    x = (np.round(rng.standard_normal((d, n)) * 200) / 200).astype(np.float32)
    x[:, :300] = x[:, :1]  # whole tiles of one point
    with Context(0) as ctx:
        ctx.set_tuning(cells_per_h3=cells3)
        a = ctx.entropy_batch([(x, [h] * d)] * few)
        pairs_few = ctx.last_stats().candidate_pairs
        assert 2432 < ctx.last_stats().tiles <= 131072  # and no tile shared out
        b = ctx.entropy_batch([(x, [h] * d)] * many)
        assert ctx.last_stats().tiles > 131072
        assert ctx.last_stats().candidate_pairs * few == pairs_few * many
    assert np.allclose(a, a[0], rtol=1e-12, atol=0) and np.allclose(b, a[0], rtol=1e-12, atol=0)
    assert abs(a[0] - O.entropy_fp64(x, [h] * d)) < 1e-6


def test_batches_launched_directly_and_through_a_graph():
    # up to 128 instances launch directly, larger batches through the context's
    # graph; calls alternate between both and between two graph shapes
    from entropical_gb300 import Context, workloads
    x = workloads.mi_coords(1500, 18, seed=4)
    h = workloads.scott_bandwidth(x, 2)
    with Context(0) as c:
        for _ in range(2):
            got = {m: c.mi_all_pairs(x[:m], h[:m])[0] for m in (15, 16, 18)}  # 120, 136, 171
        for m in (16, 18):
            assert np.max(np.abs(got[m][:15, :15] - got[15])) < 1e-9
    for i, j in [(0, 1), (3, 14)]:
        assert abs(got[18][i, j] - O.mi_fp64(x[i], x[j], h[i], h[j])) < 1e-6


def test_in_block_strip_sorts_inside_a_graph():
    # 187 densities of up to 1,200 points: captured, and the strip sorts (two
    # digits for the 3-D cells) of 176 segments run one block per segment; 40
    # densities of the same columns launch directly
    from entropical_gb300 import Context, workloads
    x = workloads.mi_coords(1200, 11, seed=9)
    h = workloads.scott_bandwidth(x, 3) * np.float32(0.3)
    with Context(0) as c:
        for _ in range(2):  # the second batch updates the graph
            all_te = c.te_all_pairs(x, h, [1])[0]
            few = c.te_all_pairs(x[:5], h[:5], [1])[0]
            assert np.max(np.abs(all_te[:5, :5] - few)) < 1e-7
    i, j = 1, 3
    assert abs(few[i, j] - O.te_fp64(x[j], x[i], 1, h[j], h[i])) < 1e-6
