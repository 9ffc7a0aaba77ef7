"""GPU: every block size that sph_batch_tune takes for the pair kernels gives
the bits of the default, and none slows the passes that stage their rows in
shared memory, whose buffers are sized for one block."""
import numpy as np
import pytest

from sph import scenes
from sph.batch import Batch

pytestmark = pytest.mark.gpu


def batch(pair_block, sizes):
    b = Batch()
    ids = [b.add(scenes.mix_member(scenes.MATERIALS[k % 3], n, seed=k, youngs_modulus=5e4, name="s%d" % k))
           for k, n in enumerate(sizes)]
    if pair_block:
        b.tune(256, pair_block, 0)
    return b, ids


@pytest.mark.parametrize("sizes", [(900, 1100, 700), (45000, 3000, 1300)])  # split over three warps; whole
def test_pair_blocks_give_the_same_bits(sizes):
    want = None
    for pair_block in (0, 32, 96, 160, 512):
        b, ids = batch(pair_block, sizes)
        b.step(3)
        got = [{f: np.array(v) for f, v in b.read(sid).items() if f in ("position", "force", "density", "stress")}
               for sid in ids]
        b.close()
        if want is None:
            want = got
        for g, w in zip(got, want):
            for f in w:
                assert np.array_equal(g[f], w[f]), (pair_block, f)


def test_staged_passes_take_no_longer_at_other_pair_blocks():
    """At most 1.15 times the default's time (the density pass took 1.9 times
    as long at blocks of 32 and of 512; repeats differ by 2%)."""
    sizes = [20000 + 1500 * k for k in range(24)]
    took = {}
    for pair_block in (128, 32, 512):
        b, _ = batch(pair_block, sizes)
        b.step(1)
        runs = [b.profile(5) for _ in range(4)]
        b.close()
        took[pair_block] = {p: min(r[p] for r in runs) for p in ("density", "corotational rotations",
                                                                 "svk deformations")}
    for pair_block in (32, 512):
        for p, ms in took[pair_block].items():
            assert ms <= 1.15 * took[128][p], (pair_block, p, took)
