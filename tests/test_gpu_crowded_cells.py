"""GPU: cells with more particles than are ordered by comparing them with
each other -- one walk over all particles' cells orders them -- against
numpy's stable sort, exactly; and what that takes."""
import time

import numpy as np
import pytest

from sph import scenes
from test_zz_no_alloc import noalloc_tables

pytestmark = pytest.mark.gpu


def piles(n, sizes, box, seed, pnum=None):
    """n particles of which sizes[q] lie in one cell each, in an order that
    has nothing to do with the cells'."""
    rng = np.random.default_rng(seed)
    h = 0.02
    pos = rng.uniform(0.0, box, size=(n, 3))
    first = 0
    for q, m in enumerate(sizes):
        pos[first:first + m] = np.array([0.31 + 2 * q, 0.31 + q % 3, 0.31]) * h + 0.4 * h * rng.random((m, 3))
        first += m
    pos = pos[rng.permutation(n)]
    sc = scenes.wcsph_block(2, 2, 2, h=h, box=(0.0, box), pnum=pnum or n, dt=1e-12)
    sc.init = {"position": pos.astype(np.float32), "n": n}
    return sc


def check(tables, n):
    cell, count, off, parts = tables
    cells = count.size
    assert np.array_equal(count, np.bincount(cell[:n], minlength=cells))
    assert np.array_equal(off, np.concatenate([[0], np.cumsum(count)[:-1]]))
    assert np.array_equal(parts[:n], np.argsort(cell[:n], kind="stable"))


# a small scene's line is above 256 + n / 256, a large one's 256 + n / 48;
# tiles of the walk hold 4,096 and 8,192 particles
@pytest.mark.parametrize("n,sizes,box", [(300, [300], 0.3), (5000, [275, 276, 277], 0.4), (8193, [400, 8193 - 400], 0.4),
                                         (16384, [320, 321] * 6, 0.7), (16384, [330] * 49, 2.0), (16384, [16384], 0.7),
                                         (17000, [610, 611, 5000], 0.7), (40961, [1109, 1110, 1111, 20000], 0.7),
                                         (100000, [9000] * 11, 1.0)])
def test_crowded_cells_in_canonical_order(n, sizes, box):
    sc = piles(n, sizes, box, seed=n + len(sizes), pnum=n + 5)
    ps = sc.system()
    names = ("gridcell", "gridcount", "celloffset", "cellparticles")
    read = lambda: [np.array(a).ravel() for a in ps.get_fields(*names)]  # noqa: E731
    ps.compute_particle_bins()
    ps.sync_device_to_host()
    named = read()
    check(named, n)
    if max(sizes) <= 20000:
        ps.update_fused(1)
        ps.sync_device_to_host()
        assert all(np.array_equal(a[:n], b[:n]) for a, b in zip(named, read()))
    res, bounds = [np.array(a) for a in ps.get_fields("gridres", "gridbounds")]
    ps.close()
    check(noalloc_tables(sc.init["position"], res, bounds)[:4], n)


def test_batch_scenes_with_crowded_cells():
    from sph.batch import Batch
    b = Batch()
    made = [piles(n, [m], 0.4, seed=n) for n, m in ((900, 600), (3000, 257), (6000, 5000))]
    ids = [b.add(sc) for sc in made]
    b.step(1)
    for sid, sc in zip(ids, made):
        got = b.read(sid)
        check([got[f].ravel() for f in ("gridcell", "gridcount", "celloffset", "cellparticles")],
              sc.init["position"].shape[0])
    b.close()


@pytest.mark.parametrize("n", [16384, 400000])
def test_a_pile_costs_no_square_of_its_size(n):
    """Ordering a pile four times as large takes less than eight times as
    long (sixteen, if every particle were compared with every other)."""
    took = []
    for m in (n // 4, n):
        ps = piles(n, [m], 0.0201 * n ** (1 / 3.0), seed=n).system()
        best = 1e9
        for _ in range(5):
            ps.synchronize()
            t0 = time.perf_counter()
            ps.compute_particle_bins()
            ps.synchronize()
            best = min(best, time.perf_counter() - t0)
        took.append(best)
        ps.close()
    # and well below the 1.1 and 24 ms that comparing took
    assert took[1] < 8 * took[0] and took[1] < n * 1e-8 + 3e-4, took
