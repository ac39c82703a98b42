"""Device decoding of XTC frames at the edges of its forms: segments of 8 to 64
atoms (chosen by frames x segments), a warp or a thread per frame's walk (256
frames per SM), the walk's batches of 128 words. Bit-exact against the oracle's
reader."""
import numpy as np
import pytest

from entropical_gb300 import write_xtc
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


# 41,000 frames and more are walked by threads (up to 160 SMs); 33 x 60000 decodes in
# 8-atom segments (of 32 atoms it would have 120,000), 129 x 90000 in 64-atom ones
@pytest.mark.parametrize("atoms,frames", [(10, 1), (10, 45000), (63, 7), (64, 7), (65, 7),
                                          (1025, 3), (70, 41000), (33, 60000),
                                          (129, 90000)])
def test_segment_forms(ctx, tmp_path, atoms, frames):
    rng = np.random.default_rng(atoms)
    base = np.cumsum(rng.normal(0, 0.12, (atoms, 3)), 0)
    # water-like triples in between: runs of small atoms of every length
    base[1::3] = base[::3][: len(base[1::3])] + 0.02
    few = min(frames, 400)
    rows = (base[None] + rng.normal(0, 0.01, (few, atoms, 3))).reshape(few, -1)
    rows = np.tile(rows, (-(-frames // few), 1))[:frames].astype(np.float32)
    p = str(tmp_path / "t.xtc")
    write_xtc(p, rows, primary="R")
    got = ctx.read_xtc(p, primary="R")
    assert got.shape == rows.shape
    ref = O.read_xtc(p) if frames <= 400 else None
    if ref is None:  # the frames repeat: check the first ones, then the repeats
        q = str(tmp_path / "few.xtc")
        write_xtc(q, rows[:few], primary="R")
        ref = np.tile(O.read_xtc(q), (-(-frames // few), 1))[:frames]
    assert np.array_equal(_bits(got), _bits(ref))
