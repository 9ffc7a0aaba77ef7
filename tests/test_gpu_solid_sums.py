"""GPU: the accuracy of a plane-free solid's force sums.

Under uniform stress on an exact lattice the pair terms of an inner particle
cancel bit for bit (the term of the partner at -x is minus that of the one
at x), so its exact elastic force is zero and what is left is the rounding
of the sum alone."""
import numpy as np
import pytest

from sph import scenes

pytestmark = pytest.mark.gpu


# In units of 2^-24 times the sum of the terms' magnitudes, emulated in
# numpy over 200 stresses and both places of a particle in its cell: one
# Kahan sum over the stencil leaves 0.08 rms, one per z plane joined with
# its compensation 0.10, one per z plane without it 0.20.
@pytest.mark.parametrize("material", ["corot", "svk"])
@pytest.mark.parametrize("dims", [(14, 14, 14), (36, 36, 33)])  # split over three warps; whole
def test_equilibrium_forces_keep_the_sums_compensation(material, dims):
    d, h = 2.0 ** -7, 2.3 * 2.0 ** -7
    sc = scenes.solid_lattice(*dims, spacing=d, h=h, material=material, clamp_layers=0)
    ps = sc.system()
    n = sc.n
    ps.set_fields(density0=np.full(n, 1000, np.float32), density=np.full(n, 1000, np.float32))
    ps.call_for_all_particles("init_original_position")
    ps.compute_particle_bins()
    mass = float(ps.get_fields("mass")[0].ravel()[0])
    o = np.stack(np.meshgrid(*[np.arange(-2, 3)] * 3), axis=-1).reshape(-1, 3) * d
    r = np.linalg.norm(o, axis=1)
    o, r = o[(r > 0) & (r <= h)], r[(r > 0) & (r <= h)]
    grad = 45.0 / (np.pi * h ** 6) * ((h - r) ** 2 / r)[:, None] * o
    left = []
    for sigma in np.random.default_rng(dims[0]).normal(size=(12, 6)).astype(np.float32) * 1e4:
        ps.set_fields(stress=np.tile(sigma, (n, 1)))
        ps.call_for_all_particles("compute_forces_solids")
        ps.sync_fields_device_to_host("force_elastic")
        fe = ps.get_fields("force_elastic")[0][:n].reshape(dims[2], dims[1], dims[0], 3)[3:-3, 3:-3, 3:-3]
        s = sigma.astype(np.float64)
        tensor = np.array([[s[0], s[3], s[4]], [s[3], s[1], s[5]], [s[4], s[5], s[2]]])
        scale = np.abs(grad @ tensor).sum(axis=0) * (mass / 1000.0) ** 2
        left.append(np.mean((fe.astype(np.float64) / scale) ** 2))
    ps.close()
    rms = np.sqrt(np.mean(left)) * 2.0 ** 24
    assert rms <= 0.14, rms
