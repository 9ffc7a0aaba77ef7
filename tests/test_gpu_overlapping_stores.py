"""GPU: several small stores in turn, whose substeps overlap on the device
(each kernel may be resident before the one ahead on its stream has ended),
give the bits of each run by itself with a wait after every substep: cell
tables, sorted copies and masks are rewritten every substep, so a read that
did not wait would show."""
import threading

import numpy as np
import pytest

from sph import scenes

pytestmark = pytest.mark.gpu

FIELDS = ("position", "velocity", "force", "density", "num_neighbours", "gridcount", "celloffset", "cellparticles")
STEPS = 60


def make():
    out = []
    for k in range(4):
        sc = scenes.wcsph_block(8 + 2 * k, 9, 10, jitter=8e-4, seed=k, dt=2e-4)
        rng = np.random.default_rng(k)
        sc.init = dict(sc.init, velocity=rng.normal(0, 0.5, (sc.n, 3)).astype(np.float32))
        out.append(sc)
    for k, m in enumerate(("corot", "svk", "corot")):
        out.append(scenes.solid_lattice(6 + k, 7, 11, material=m, youngs_modulus=5e4, jitter=2e-4, seed=k,
                                        clamp_layers=1))
    return out


def store(sc):
    ps = sc.system()
    if sc.material != "fluid":
        ps.call_for_all_particles("init_original_position")
        ps.compute_particle_bins()
        ps.call_for_all_particles("compute_original_density")
    return ps


def result(ps):
    ps.sync_device_to_host()
    return [np.array(a) for a in ps.get_fields(*FIELDS)]


def same(got, want):
    for k, (g, w) in enumerate(zip(got, want)):
        for f, a, b in zip(FIELDS, g, w):
            assert np.array_equal(a, b), (k, f)


def waited():
    out = []
    for sc in make():
        ps = store(sc)
        for _ in range(STEPS):
            ps.update_fused(1)
            ps.synchronize()
        out.append(result(ps))
        ps.close()
    return out


def test_stores_in_turn_equal_each_alone():
    want = waited()
    all_ps = [store(sc) for sc in make()]
    for _ in range(STEPS):
        for ps in all_ps:
            ps.update_fused(1)
    same([result(ps) for ps in all_ps], want)
    for ps in all_ps:
        ps.close()


def test_stores_of_several_threads_equal_each_alone():
    want = waited()
    all_ps = [store(sc) for sc in make()]

    def run(ps):
        for _ in range(STEPS // 10):
            ps.update_fused(10)

    ts = [threading.Thread(target=run, args=(ps,)) for ps in all_ps]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    same([result(ps) for ps in all_ps], want)
    for ps in all_ps:
        ps.close()
