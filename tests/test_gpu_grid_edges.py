"""GPU: the neighbour grid at the edges of its kernels, against the oracle,
exactly: cells of one particle up to thousands, particles in an order that
has nothing to do with the cells', grids of one cell, of several scan tiles
and of more tiles than the binning counts in shared memory, and fewer
active particles than a block."""
import numpy as np
import pytest

from helpers import oracle_of
from sph import scenes

pytestmark = pytest.mark.gpu


def scene(n, box, h, crowd, seed):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0.0, box, size=(n, 3))
    k = min(crowd, n)
    pos[:k] = 0.31 * h + 0.5 * h * rng.random((k, 3))  # one cell
    pos = pos[rng.permutation(n)]
    sc = scenes.wcsph_block(2, 2, 2, h=h, box=(0.0, box), pnum=n + 3)
    sc.init = {"position": pos.astype(np.float32), "n": n}
    return sc


@pytest.mark.parametrize("n,box,h,crowd", [(1, 0.02, 0.02, 1), (255, 0.02, 0.02, 255), (2000, 0.4, 0.02, 33),
                                           (5000, 0.4, 0.02, 3000), (40000, 0.7, 0.02, 40), (70000, 1.0, 0.02, 500),
                                           (3000, 1.3, 0.01, 64)])
def test_grid_matches_oracle(n, box, h, crowd):
    sc = scene(n, box, h, crowd, seed=n)
    ps = sc.system()
    o = oracle_of(ps)
    o.call("compute_particle_bins")
    names = ("gridcell", "gridcount", "celloffset", "cellparticles")
    ps.compute_particle_bins()
    ps.sync_device_to_host()
    for f in names:
        got, want = ps.get_fields(f)[0].ravel(), o.a[f].ravel()
        m = n if f in ("gridcell", "cellparticles") else got.size
        assert np.array_equal(got[:m], want[:m]), f
    tables = [np.array(a) for a in ps.get_fields(*names)]
    ps.update_fused(1)  # the same tables from a substep's binning
    ps.sync_device_to_host()
    for f, a, b in zip(names, tables, ps.get_fields(*names)):
        m = n if f in ("gridcell", "cellparticles") else a.size
        assert np.array_equal(a.ravel()[:m], b.ravel()[:m]), f
    ps.close()


@pytest.mark.parametrize("n,cells_side", [(1, 1), (511, 7), (4096, 40), (4097, 40), (16384, 39), (16384, 41)])
def test_small_scene_grid_at_its_limits(n, cells_side):
    """One to four particles a thread, the last size before the launches of
    a large scene (pnum 16,384 with 39^3 cells) and a grid past the line."""
    rng = np.random.default_rng(n)
    h = 0.02
    box = cells_side * h + 1e-4
    sc = scenes.wcsph_block(2, 2, 2, h=h, box=(0.0, box), pnum=n)
    pos = rng.uniform(-0.01, box + 0.01, size=(n, 3))  # some outside
    sc.init = {"position": pos.astype(np.float32), "n": n}
    ps = sc.system()
    o = oracle_of(ps)
    o.call("compute_particle_bins")
    ps.compute_particle_bins()
    ps.sync_device_to_host()
    for f in ("gridcell", "gridcount", "celloffset", "cellparticles"):
        assert np.array_equal(ps.get_fields(f)[0].ravel(), o.a[f].ravel()), f
    ps.close()
