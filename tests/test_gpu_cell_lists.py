"""The device sort and tile plan at the sizes where their forms change: radix
chunks of 2,048 values, segments whose scatter blocks sum their own histogram
rows (small sorts) or read a prefix kernel's, and non-finite input anywhere in
a column."""
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


@pytest.mark.parametrize("n", [1, 31, CHUNK - 1, CHUNK, CHUNK + 1, 3 * CHUNK + 5,
                               256 * CHUNK, 256 * CHUNK + 1])
def test_sort_at_chunk_edges(ctx, n):
    # 256 chunks: the largest column whose scatter blocks sum the rows themselves
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
