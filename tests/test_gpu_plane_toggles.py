"""GPU: symmetry planes that are set and cleared between substeps.  Which
variant of the pair passes runs is decided on the device by the planes of the
moment, and with it who sums the density, applies the stress law and steps
the particles: fused (one captured graph throughout), by name and in a batch,
each stage against a store made from the same state, bit for bit, and against
the oracle.  A stale decision would skip the scene or step it twice."""
import numpy as np
import pytest

from helpers import oracle_of, rel_err
from sph import scenes
from sph.batch import Batch

pytestmark = pytest.mark.gpu

MATERIALS = ("fluid", "corot", "svk")
STEPS = 2
STAGES = ([], [0], [], [0, 2], [1])  # the planes set in each
NAMED = {"fluid": ("compute_density", "compute_forces_fluids", "step_forward"),
         "corot": ("compute_density", "compute_rotations_and_strains", "compute_stresses", "compute_forces_solids",
                   "step_forward"),
         "svk": ("compute_density", "compute_deformations", "compute_stresses", "compute_forces_solids",
                 "step_forward")}


def scene(material, seed=3):
    if material == "fluid":
        sc = scenes.wcsph_block(9, 7, 8, spacing=0.01, h=0.02, box=(-0.1, 0.4), jitter=5e-4, seed=seed, dt=1e-4)
    else:
        sc = scenes.solid_lattice(7, 6, 9, material=material, youngs_modulus=2e4, jitter=2e-4, seed=seed,
                                  clamp_layers=1)
    sc.entries = [("symmetry_planes", "3, 2, 3", "float", None) if e[0] == "symmetry_planes" else e
                  for e in sc.entries]
    rng = np.random.default_rng(seed)
    sc.init = dict(sc.init, velocity=rng.normal(0, 0.05, (sc.n, 3)).astype(np.float32))
    return sc


def planes(which):
    p = np.zeros((3, 2, 3), np.float32)
    for a in which:
        p[a, 1, a] = 1.0
    return p


def setup(ps, material):
    if material != "fluid":
        ps.call_for_all_particles("init_original_position")
        ps.compute_particle_bins()
        ps.call_for_all_particles("compute_original_density")


def run(ps, material, named):
    for _ in range(STEPS):
        if not named:
            ps.update_fused(1)
            continue
        ps.compute_particle_bins()
        for call in NAMED[material]:
            ps.call_for_all_particles(call)


def state(ps, sc):
    ps.sync_device_to_host()
    return {e[0]: np.array(ps.get_fields(e[0])[0]) for e in sc.entries if ps.get_fields(e[0])[0].size}


@pytest.mark.parametrize("material", MATERIALS)
@pytest.mark.parametrize("named", [False, True])
def test_planes_set_and_cleared_between_substeps(material, named):
    sc = scene(material)
    ps = sc.system()
    setup(ps, material)
    for which in STAGES:
        ps.set_fields(symmetry_planes=planes(which))
        before = state(ps, sc)
        orc = oracle_of(ps)
        run(ps, material, named)
        after = state(ps, sc)
        fresh = sc.system()
        fresh.set_fields(True, **before)
        fresh.sync_host_to_device()
        run(fresh, material, named)
        for f, a in state(fresh, sc).items():
            assert np.array_equal(a, after[f]), (which, f)
        fresh.close()
        orc.run(material, STEPS)
        n = sc.n
        assert rel_err(after["position"][:n], orc.a["position"][:n]) <= 1e-5
        # what the stage added to the velocities: half of it if a substep
        # were skipped
        added = [np.asarray(v, np.float64) - before["velocity"][:n] for v in (after["velocity"][:n],
                                                                              orc.a["velocity"][:n])]
        assert rel_err(*added) <= 1e-3, which
    ps.close()


@pytest.mark.parametrize("large", [False, True])  # split over three warps; whole
def test_planes_set_and_cleared_in_a_batch(large):
    made = [scene(m, seed=5) for m in MATERIALS]
    never = [scenes.solid_lattice(5, 5, 7, material="svk", youngs_modulus=5e4, jitter=1e-4, seed=4, clamp_layers=1),
             scenes.wcsph_block(36, 36, 36, jitter=1e-4, seed=2) if large else scenes.wcsph_block(6, 6, 6, seed=2)]
    alone = []
    for sc in made:
        ps = sc.system()
        setup(ps, sc.material)
        alone.append(ps)
    b = Batch()
    ids = [b.add(sc) for sc in made]
    for sc in never:
        b.add(sc)
    for which in STAGES:
        for ps, sid in zip(alone, ids):
            ps.set_fields(symmetry_planes=planes(which))
            b.scenes[sid].views["symmetry_planes"][...] = planes(which)
        b.write_fields_async(ids, "symmetry_planes")
        b.step(STEPS)
        for ps, sid, sc in zip(alone, ids, made):
            ps.update_fused(STEPS)
            want, got = state(ps, sc), b.read(sid)
            for f in ("position", "velocity", "force", "density", "num_neighbours", "symmetry_planes"):
                assert np.array_equal(got[f], want[f]), (which, sc.material, f)
    b.close()
    for ps in alone:
        ps.close()
