"""Batches on both sides of the lines between the two forms of the tile plan, lanes
per slot and a thread per slot: 16,384 slots, 8,192 per run around a tile (12,288 more
for up to 128 instances, which launch directly), 65,536 for batches with a work list.
The same tiles and runs, so the same sums up to the order of the FP64 additions."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,h,cells3,body,line", [
    (1, 0.3, 1, None, 16384),        # one run
    (2, 0.3, 1, 4, 5 * 8192),        # five
    (2, 1e-3, 1, 4, 5 * 8192 + 12288),  # runs joined over strips of a few points
    (3, 0.3, 1, None, 9 * 8192),     # nine
    (3, 1e-3, 1, None, 9 * 8192 + 12288),
    (3, 0.3, 2, None, 131072),       # 25: by 32 lanes
    (2, 0.3, 1, 7, 65536),           # strip moments, with a work list
])
def test_either_side(d, h, cells3, body, line):
    from entropical_gb300 import Context
    rng = np.random.default_rng(11 * d)
    n = 2500
    x = (np.round(rng.standard_normal((d, n)) * 200) / 200).astype(np.float32)
    x[:, :300] = x[:, :1]  # whole tiles of one point
    with Context(0) as c:
        c.set_tuning(cells_per_h3=cells3, pair_variant=[None, body, None])
        c.entropy_batch([(x, [h] * d)] * 150)  # enough tiles that none is shared out
        assert c.last_stats().tiles % 150 == 0
        each = c.last_stats().tiles // 150
        got, pairs = {}, {}
        # launched directly or as a graph (the cap of 131,072 is the same for both)
        assert line == 131072 or (line // each + 1 <= 128) == (h < 0.1)
        for k in (line // each, line // each + 1):
            got[k] = c.entropy_batch([(x, [h] * d)] * k)
            s = c.last_stats()
            assert s.tiles == k * each
            assert s.candidate_pairs % k == 0
            pairs[k] = s.candidate_pairs // k
    (a, b), (pa, pb) = got.values(), pairs.values()
    assert pa == pb
    assert np.allclose(a, a[0], rtol=1e-12, atol=0) and np.allclose(b, a[0], rtol=1e-12, atol=0)
    assert abs(a[0] - O.entropy_fp64(x, [h] * d)) < 1e-6
