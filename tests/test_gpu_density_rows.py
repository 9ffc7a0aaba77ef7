"""GPU: the density pass's staged rows at their edges, against the oracle:
rows shorter and longer than a 32-candidate chunk and than 64 candidates,
starts at every offset from a multiple of four, planes of rows wider than
the staging buffer (a direct walk), a block of one particle, and pairs at
the bound itself.  Neighbour counts are bit-exact; densities within 1e-5 of
the largest, the bound of the other density tests."""
import numpy as np
import pytest

from helpers import max_rel, oracle_of
from sph import scenes

pytestmark = pytest.mark.gpu


def cloud(n, per_cell, seed, on_lattice=False):
    """n particles at about per_cell in each cell of side h = 0.02."""
    rng = np.random.default_rng(seed)
    side = 0.02 * (n / per_cell) ** (1.0 / 3.0)
    pos = 0.11 + side * rng.random((n, 3))
    if on_lattice:  # distances of exactly h along the axes, up to rounding
        pos = np.round(pos / 0.01) * 0.01 + rng.integers(-1, 2, size=(n, 3)) * 2.0 ** -26
    sc = scenes.wcsph_block(2, 2, 2, box=(0.0, 0.4), pnum=n + 5)
    sc.init = {"position": pos.astype(np.float32), "n": n}
    return sc


@pytest.mark.parametrize("n,per_cell,lattice", [(1, 8, False), (33, 0.3, False), (129, 2, False), (700, 8, True),
                                                (1000, 11, False), (1500, 22, False), (2500, 40, False),
                                                (4000, 130, False)])
def test_density_rows_match_oracle(n, per_cell, lattice):
    for seed in range(4):  # the starts' offsets within four differ
        sc = cloud(n - seed if n > 8 else n, per_cell, seed, lattice)
        m = sc.init["position"].shape[0]
        ps = sc.system()
        o = oracle_of(ps)
        for call in ("compute_particle_bins", "compute_density"):
            o.call(call)
        # the named pass, and the one of a fused substep (which records
        # the masks that the forces then walk)
        ps.compute_particle_bins()
        ps.call_for_all_particles("compute_density")
        ps.sync_device_to_host()
        count, dens = (np.array(a[:m]) for a in ps.get_fields("num_neighbours", "density"))
        assert np.array_equal(count, o.a["num_neighbours"][:m])
        assert max_rel(dens, o.a["density"][:m]) <= 1e-5
        ps.update_fused(1)
        ps.sync_device_to_host()
        fused = ps.get_fields("num_neighbours", "density")
        assert np.array_equal(fused[0][:m], count) and np.array_equal(fused[1][:m], dens)
        ps.close()


def test_split_and_whole_passes_give_the_same_bits():
    """A scene alone (its stencils split over three warps) and in a batch
    whose particles are past the line (whole): the same bits, with rows of
    every length, a cell above 64 candidates a row and spare capacity."""
    from sph.batch import Batch
    for n, per_cell in ((1, 8), (31, 3), (700, 8), (1500, 22), (2500, 60)):
        sc = cloud(n, per_cell, n)
        ps = sc.system()
        ps.update_fused(3)
        ps.sync_device_to_host()
        b = Batch()
        sid = b.add(sc)
        b.add(scenes.wcsph_block(36, 36, 36, jitter=1e-4, seed=2))
        b.step(3)
        got = b.read(sid)
        for f in ("position", "velocity", "force", "density", "num_neighbours"):
            assert np.array_equal(got[f], ps.get_fields(f)[0]), f
        b.close()
        ps.close()
