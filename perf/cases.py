"""The work that programs have this framework do, as cases that can be timed
and compared: one or a few substeps of a WCSPH fluid, of a corotational or
St. Venant-Kirchhoff solid, of an interacting fluid-solid scene and of a
batch of uneven scenes, through the calls such programs make.

A pass is one iteration of the program's loop.  It leaves its results where
that loop finds them: in the store's fields on the device (returned as
views of them), or, where the loop reads them back, in the host store.
Passes follow each other on the same state, as substeps do.  Where a case
is small enough to be run thousands of times, its time step is 1e-6 s
rather than the configuration's, so that the scene stays in the state that
the case stands for; the work of a substep does not depend on it.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "opencl-sph_gb300"))
from sph import bindings as bnd  # noqa: E402
from sph import scenes  # noqa: E402
from sph.batch import Batch  # noqa: E402
from sph.systems import FluidSystem, ParticleSystem, StrainSolid, SVKSolid  # noqa: E402

FLUID_FIELDS = ("position", "velocity", "acceleration", "force", "density", "num_neighbours", "gridcell",
                "gridcount", "celloffset", "cellparticles")
SOLID_FIELDS = FLUID_FIELDS + ("stress", "force_elastic", "force_viscous", "cutoff_force")
FIELDS = {"fluid": FLUID_FIELDS, "corot": SOLID_FIELDS + ("rotation", "strain"),
          "svk": SOLID_FIELDS + ("deformation",), "mixed": SOLID_FIELDS + ("deformation",)}
NAMED = {"fluid": FluidSystem, "corot": StrainSolid, "svk": SVKSolid}
BAR_FIELDS = ("position", "velocity", "strain", "stress", "force")
BATCH_STEPS = 5


def listed():
    def fluid(name, nx, ny, nz, **kw):
        return dict({"name": name, "kind": "fluid", "nx": nx, "ny": ny, "nz": nz, "api": "fused", "steps": 1,
                     "dt": 1e-6, "jitter": 0.01, "mixed_up": False, "spare": 0}, **kw)

    def solid(name, kind, nx, ny, nz, **kw):
        return dict({"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "api": "fused", "steps": 1,
                     "dt": 1e-6, "jitter": 0.01}, **kw)

    return [
        # the smallest scene of the batched mix on its own, ragged, one
        # substep a call: launches and latency
        fluid("fluid-1k", 11, 7, 13),
        # the dam break (20^3), ten substeps a call as between two frames
        fluid("fluid-8k x10", 20, 20, 20, steps=10),
        # the same scene through the reference driver's loop: the kernels
        # called by name, one by one
        fluid("fluid-8k named", 20, 20, 20, api="named"),
        # a flow that has run for a while: no lattice left, particle order
        # no longer the cells' order, a store with spare capacity
        fluid("fluid-100k settled", 53, 31, 61, jitter=0.1, mixed_up=True, spare=777),
        # the million-particle slab
        fluid("fluid-1m", 128, 64, 128, dt=2e-5),
        # the corotational beam (10 x 10 x 40)
        solid("corot-4k", "corot", 10, 10, 40),
        # the largest corotational scene of the batched mix
        solid("corot-65k", "corot", 32, 32, 64),
        # the 32^3 St. Venant-Kirchhoff cube
        solid("svk-32k", "svk", 32, 32, 32),
        # a small St. Venant-Kirchhoff beam by the reference driver's loop
        solid("svk-1k5 named", "svk", 9, 9, 19, api="named"),
        # the reference's strain test: a bar between two constraint planes,
        # which its loop moves, with the store of the solid conf (its slots
        # for symmetry planes unset) and results read back every substep
        {"name": "strain bar", "kind": "bar", "nx": 21, "ny": 9, "nz": 9, "dt": 1e-6, "jitter": 0.01},
        # fluid, an elastic cube and a rigid ball in one scene: the large
        # configuration
        {"name": "mixed-1m", "kind": "mixed", "nx": 128, "ny": 64, "nz": 128, "cube": 32, "ball": 10.0,
         "dt": 2e-5, "jitter": 0.01},
        # a batch of uneven scenes, 60% fluid, 25% corotational, 15% SVK,
        # a few substeps between two reads of every position
        {"name": "batch-64", "kind": "batch", "count": 64, "lo": 1000, "hi": 65536, "sizes": 0, "dt": 1e-4, "jitter": 0.01},
    ]


def _draw_dims(rng, lo, hi):
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    ax, ay = math.exp(rng.uniform(-0.5, 0.5)), math.exp(rng.uniform(-0.5, 0.5))
    s = (n / (ax * ay)) ** (1.0 / 3.0)
    return {"nx": max(3, round(ax * s)), "ny": max(3, round(ay * s)), "nz": max(3, round(s))}


def draw(rng):
    kind = rng.choices(("fluid", "corot", "svk", "bar", "mixed", "batch"), (8, 4, 3, 1, 2, 2))[0]
    case = {"kind": kind, "dt": 1e-6, "jitter": rng.choice((0.01, 0.03, 0.1))}
    if kind == "fluid":
        case.update(_draw_dims(rng, 500, 700000))
        case.update({"api": rng.choice(("fused", "fused", "named")), "steps": rng.choice((1, 1, 2, 5)),
                     "mixed_up": rng.random() < 0.5, "spare": rng.choice((0, 0, rng.randrange(1, 2000)))})
        if case["nx"] * case["ny"] * case["nz"] > 150000:
            case["steps"] = 1
    elif kind in ("corot", "svk"):
        case.update(_draw_dims(rng, 500, 100000))
        case.update({"api": rng.choice(("fused", "fused", "named")), "steps": 1,
                     "jitter": min(case["jitter"], 0.03)})
    elif kind == "bar":
        case.update(_draw_dims(rng, 500, 4096))
        case["jitter"] = min(case["jitter"], 0.03)
    elif kind == "mixed":
        case.update(_draw_dims(rng, 20000, 400000))
        case["cube"] = rng.randrange(6, max(7, min(case["nx"], case["nz"]) // 2))
        case["ball"] = rng.uniform(3.0, max(3.5, 0.2 * min(case["nx"], case["nz"])))
        case["jitter"] = 0.01
    else:
        case.update({"count": rng.randrange(3, 65), "lo": 1000, "hi": rng.choice((8000, 20000, 40000)),
                     "sizes": rng.randrange(1000),
                     "dt": 1e-4, "jitter": 0.01})
    return case


# ---- inputs ---------------------------------------------------------------------

def _flow(pos, scale, rng, speed, noise):
    """A smooth velocity field with a little noise."""
    k = 2.0 * math.pi / scale
    x, y, z = (pos[:, a].astype(np.float64) for a in range(3))
    v = speed * np.stack([np.sin(k * y) * np.cos(k * z), np.sin(k * z) * np.cos(k * x),
                          np.sin(k * x) * np.cos(k * y)], axis=1)
    return (v + rng.uniform(-noise, noise, size=v.shape)).astype(np.float32)


def _scene(case, seed):
    """(scene, fields set after a solid's rest state has been recorded)."""
    rng = np.random.default_rng([7, int(seed)])
    kind = case["kind"]
    if kind == "fluid":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        n = nx * ny * nz
        slab = n > 1000000
        d = 0.005 if slab else 0.01
        # a box twice the block's width, room to collapse
        hi = 1.0 if slab else round(2 * max(nx, ny, nz) * d + 0.08, 6)
        sc = scenes.wcsph_block(nx, ny, nz, spacing=d, h=2 * d, box=(0.0, hi), jitter=case["jitter"] * d,
                                seed=int(seed), dt=case["dt"], pnum=n + case["spare"],
                                **({"stiffness": 0.375, "viscosity": 0.025} if slab else {}))
        pos = sc.init["position"]
        if case["mixed_up"]:
            pos = pos[rng.permutation(n)]
        sc.init["position"] = pos
        sc.init["velocity"] = _flow(pos, hi, rng, 0.2, 0.02)
        return sc, {}
    if kind == "mixed":
        d = 0.005
        hi = round(max(1.0, 0.0055 * max(case["nx"], case["nz"], case["ny"] + case["cube"] + 2 * case["ball"] + 8)), 6)
        # the cube rests on the fluid, the ball falls beside it from above
        r = case["ball"] * d
        top = (case["ny"] + case["cube"]) * d
        ball = (r, (r + 3 * d, top + r + 2 * d, r + 3 * d), (0.0, -0.1, 0.0))
        sc = scenes.fluid_solid_scene(fluid=(case["nx"], case["ny"], case["nz"]), cube=(case["cube"],) * 3, ball=ball,
                                      spacing=d, h=2 * d, box=(0.0, hi), stiffness=0.375, viscosity=0.025,
                                      dt=case["dt"], jitter=case["jitter"] * d, seed=int(seed))
        return sc, {}
    sc = scenes.solid_lattice(case["nx"], case["ny"], case["nz"], material="corot" if kind == "bar" else kind,
                              youngs_modulus=5e4, poisson=0.35 if kind == "svk" else 0.3, dt=case["dt"],
                              clamp_layers=0 if kind == "bar" else 1, jitter=case["jitter"] * 0.01, seed=int(seed),
                              gravity=(0.0, 0.0, 0.0) if kind == "bar" else (0.0, -9.8, 0.0))
    x0 = sc.init["position"]
    x = x0.astype(np.float64)
    length = x[:, 2].max()
    # a beam bent downwards, 1% stretched
    x[:, 1] -= 0.08 * length * (x[:, 2] / length) ** 2
    x[:, 2] *= 1.01
    x += rng.uniform(-1e-5, 1e-5, size=x.shape)
    later = {"position": x.astype(np.float32), "velocity": _flow(x0, length, rng, 0.05, 0.005)}
    if kind == "bar":
        sizes = {"plane_constraints": "3, 2, 4", "symmetry_planes": "3, 2, 3"}
        sc.entries = [(e[0], sizes.get(e[0], e[1]), e[2], e[3]) for e in sc.entries]
        on = np.zeros(sc.n, np.uint32)
        on[x0[:, 0] < 0.005] = 1
        on[x0[:, 0] > (case["nx"] - 1.5) * 0.01] = 2
        sc.init["plane_constraints_particles"] = on
    return sc, later


def _batch_scenes(case, seed):
    rng = np.random.default_rng([11, case["sizes"]])  # the requests; the seed gives each its particles
    jitters = np.random.default_rng([13, int(seed)])
    out = []
    for k in range(case["count"]):
        n = math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))
        kind = scenes.MATERIALS[int(rng.choice(3, p=(0.6, 0.25, 0.15)))]
        e = math.exp(rng.uniform(math.log(1e4), math.log(1e6 if kind == "corot" else 1e5)))
        out.append(scenes.mix_member(kind, n, seed=int(jitters.integers(1 << 30)), youngs_modulus=e,
                                     poisson=rng.uniform(0.25, 0.45), dt_fluid=case["dt"], dt_solid=0.5 * case["dt"],
                                     jitter=case["jitter"] * 0.01, name="s%02d" % k))
    return out


class _Held(object):
    """A system or a batch, closed when nothing refers to it any more."""

    def __init__(self, what):
        self.what = what

    def __del__(self):
        self.what.close()


class _Device(object):
    """A field of a device store for torch.as_tensor (no copy); the view
    keeps the store."""

    def __init__(self, address, shape, kind, held):
        self.held = held
        self.__cuda_array_interface__ = {"data": (address, False), "shape": shape, "typestr": kind, "version": 3,
                                         "strides": None}


class _Host(object):
    """A field of a host store for numpy.asarray (no copy); the view keeps
    the store."""

    def __init__(self, view, held):
        self.held = held
        self.__array_interface__ = dict(view.__array_interface__)


class _State(object):
    """What a program keeps between its passes."""

    def __init__(self, case):
        self.case = case


def prepare(case, seed):
    s = _State(case)
    kind = case["kind"]
    if kind == "batch":
        s.batch = Batch()
        held = _Held(s.batch)
        s.ids = [s.batch.add(sc) for sc in _batch_scenes(case, seed)]
        for sid in s.ids:
            s.batch.pin(sid)
        s.out = [np.asarray(_Host(s.batch.scenes[sid].views["position"], held)) for sid in s.ids]
        return s
    sc, later = _scene(case, seed)
    if case.get("api") == "named" or kind == "bar":
        cls = NAMED["corot" if kind == "bar" else kind]
    else:
        cls = ParticleSystem
    ps = s.system = cls(spec=sc.spec, kernel_files=sc.kernel_files)
    held = _Held(ps)
    ps.set_fields(True, **sc.init)
    ps.sync_host_to_device()
    if kind != "fluid":
        # a solid's rest state, as StrainSolid.setup() records it
        ps.call_for_all_particles("init_original_position")
        ps.compute_particle_bins()
        ps.call_for_all_particles("compute_original_density")
    if later:
        ps.set_fields(**later)
    if kind == "bar":
        x0 = sc.init["position"]
        planes = np.zeros((4, 2, 3), np.float32)
        planes[0, 0, 0], planes[0, 1, 0] = -1e-4, 1.0
        planes[1, 0, 0], planes[1, 1, 0] = float(x0[:, 0].max()) + 1e-4, 1.0
        s.planes = planes
        s.out = {k: np.asarray(_Host(ps.get_fields(k)[0][: sc.n], held)) for k in BAR_FIELDS}
        ps.synchronize()
        return s
    base = ps.psdata_opencl.data
    s.out = {}
    for name in FIELDS[kind]:
        f = bnd.get_field_psdata(ps.psdata, name)
        view = ps.get_fields(name)[0]
        per_particle = view.shape[0] == sc.n + case.get("spare", 0) and not name.startswith(("gridcount", "cello"))
        shape = (sc.n,) + view.shape[1:] if per_particle else view.shape
        kind_ = "<f4" if view.dtype == np.float32 else "<i4"
        s.out[name] = torch.as_tensor(_Device(base + ps.psdata.data_offsets[f], shape, kind_, held), device="cuda")
    ps.synchronize()
    return s


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "batch":
        s.batch.step(BATCH_STEPS)
        s.batch.read_fields(s.ids, "position")
        return s.out
    ps = s.system
    if kind == "bar":
        ps.set_fields(True, plane_constraints=s.planes)
        ps.sync_fields_host_to_device("plane_constraints")
        ps.update()
        ps.call_for_all_particles("apply_plane_constraints")
        ps.sync_fields_device_to_host(*BAR_FIELDS)
        return s.out
    if case.get("api") == "named":
        for _ in range(case["steps"]):
            ps.update()
    else:
        ps.update_fused(case.get("steps", 1))
    return s.out


# ---- what a pass cannot do without ------------------------------------------------

def work(case):
    """Bytes: each particle's state read once and its results written once,
    and the cell tables written.  Operations: about 34 neighbours a particle
    within h (spacing h / 2), with the pair terms of density and forces."""
    kind = case["kind"]
    if kind == "batch":
        n = case["count"] * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        return {"bytes": BATCH_STEPS * n * (2 * 24 + 60 + 8 + 0.4 * 200) + 12 * n, "flops": BATCH_STEPS * n * 34 * 60}
    n = case["nx"] * case["ny"] * case["nz"]
    steps = case.get("steps", 1)
    if kind in ("corot", "svk", "bar"):
        # + rest position, density0, body; rotation or deformation, strain,
        # stress and the three parts of the force
        return {"bytes": steps * n * (24 + 24 + 32 + 20 + 136 + 8), "flops": steps * n * 34 * 150}
    # position, velocity in; position, velocity, acceleration, force, density,
    # count out; cell and order out; 2 words a cell
    return {"bytes": steps * n * (24 + 24 + 32 + 8 + 8), "flops": steps * n * 34 * 60}


# ---- 64-bit results ----------------------------------------------------------------

PI = 3.14159265358979323846


def _f64(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda" if torch.cuda.is_available() else "cpu").double()


def _pairs(x, h):
    """All ordered pairs (i, j), j != i, with |x_j - x_i| <= h."""
    cell = ((x - x.min(0).values) / h).floor().long()
    dims = (cell.max(0).values + 3).tolist()
    cell = cell + 1
    key = (cell[:, 2] * dims[1] + cell[:, 1]) * dims[0] + cell[:, 0]
    order = torch.argsort(key)
    sk = key[order]
    ids = torch.arange(x.shape[0], device=x.device)
    found_i, found_j = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            # the three cells of a row are one range
            k = (dz * dims[1] + dy) * dims[0] + key
            b = torch.searchsorted(sk, k - 1, right=False)
            m = torch.searchsorted(sk, k + 1, right=True) - b
            for t in range(int(m.max())):
                live = ids[m > t]
                j = order[b[live] + t]
                near = ((x[j] - x[live]) ** 2).sum(1) <= h * h
                near &= j != live
                found_i.append(live[near])
                found_j.append(j[near])
    return torch.cat(found_i), torch.cat(found_j)


def _sum(n, i, v):
    return torch.zeros((n,) + v.shape[1:], dtype=v.dtype, device=v.device).index_add_(0, i, v)


def _param(sc, name):
    return float(np.float32(sc.param(name)))


def _density(x, i, j, h, mass):
    w = (h * h - ((x[j] - x[i]) ** 2).sum(1)).clamp_min(0) ** 3
    own = torch.full((x.shape[0],), (h * h) ** 3, dtype=x.dtype, device=x.device)
    return (_sum(x.shape[0], i, w) + own) * mass * 315.0 / (64.0 * PI * h ** 9)


def _grad(d, h):
    """The spiky kernel's gradient at d, zero beyond h."""
    r = d.norm(dim=1)
    s = torch.where((r <= h) & (r > 0), -45.0 / (PI * h ** 6) * (h - r) ** 2 / r.clamp_min(1e-300), torch.zeros_like(r))
    return d * s[:, None]


def _fluid_force(sc, x, v, rho, i, j, phase=None):
    h, mass = _param(sc, "smoothingradius"), _param(sc, "mass")
    p = (rho - _param(sc, "restdens")) * _param(sc, "stiffness")
    pi, pj = p[i], p[j]
    if phase is not None:
        solid = (phase[i] + phase[j]) > 0
        both = (phase[i] * phase[j]) > 0
        pi, pj = (torch.where(solid, q.clamp_min(0), q) for q in (pi, pj))
    d = x[j] - x[i]
    r = d.norm(dim=1)
    kv = 45.0 / (PI * h ** 6)
    pt = -0.5 * (pi + pj) * kv * (h - r) ** 2 / r.clamp_min(1e-300)
    f = (d * pt[:, None] + (v[j] - v[i]) * (_param(sc, "viscosity") * kv * (h - r))[:, None]) / (rho[i] * rho[j])[:, None]
    if phase is not None:
        f = torch.where(both[:, None], torch.zeros_like(f), f)
    return _sum(x.shape[0], i, f) * mass


def _polar(a):
    a = a * (math.sqrt(3.0) / a.flatten(1).norm(dim=1))[:, None, None]
    for _ in range(12):
        a = 0.5 * (a + torch.linalg.inv(a).transpose(1, 2))
    return a


def _sym(m):
    return torch.stack([m[:, 0, 0], m[:, 1, 1], m[:, 2, 2], 0.5 * (m[:, 0, 1] + m[:, 1, 0]),
                        0.5 * (m[:, 0, 2] + m[:, 2, 0]), 0.5 * (m[:, 1, 2] + m[:, 2, 1])], dim=1)


def _stencil(sc, x, i, j):
    """Whether j lies in the 27 cells around i's."""
    gb = np.float32(sc.param("gridbounds")).reshape(3, 2)
    res = np.floor(np.abs((gb[:, 1] - gb[:, 0]).astype(np.float64)) / _param(sc, "smoothingradius"))
    lo, ext, r = _f64(gb[:, 0]), _f64(gb[:, 1]) - _f64(gb[:, 0]), _f64(res)
    c = torch.minimum(((x - lo) / ext * r).floor().clamp_min(0), r - 1)
    return ((c[j] - c[i]).abs() <= 1).all(1)


def _solid(sc, x, v, x0, body, soft, svk):
    """rotation or deformation, strain, stress and forces of a solid; `soft`
    are its particles (a mixed scene's solid phase)."""
    n, dev = x.shape[0], x.device
    h, mass = _param(sc, "smoothingradius"), _param(sc, "mass")
    e, nu = _param(sc, "youngs_modulus"), _param(sc, "poisson")
    i, j = _pairs(x, h)
    rho = _density(x, i, j, h, mass)
    keep = soft[i] & soft[j]
    i, j = i[keep], j[keep]
    i0, j0 = _pairs(x0, h)
    keep = soft[i0] & soft[j0]
    rho0 = _density(x0, i0[keep], j0[keep], h, mass)
    keep &= _stencil(sc, x, i0, j0)
    i0, j0 = i0[keep], j0[keep]
    p, q = x[j] - x[i], x0[j] - x0[i]
    w = (h * h - (p ** 2).sum(1)).clamp_min(0) ** 3
    apq = _sum(n, i, (p * w[:, None])[:, :, None] * q[:, None, :])
    eye = torch.eye(3, dtype=x.dtype, device=dev).expand(n, 3, 3)
    out = {}
    lam, mu2 = e * nu / (1 + nu) / (1 - 2 * nu), e / (1 + nu)
    full = lambda s: torch.stack([s[:, 0], s[:, 3], s[:, 4], s[:, 3], s[:, 1], s[:, 5], s[:, 4], s[:, 5], s[:, 2]],  # noqa: E731
                                 dim=1).reshape(-1, 3, 3)
    if svk:
        aqq = _sum(n, i, (q * w[:, None])[:, :, None] * q[:, None, :])
        alone = aqq.flatten(1).abs().amax(1) == 0
        f = apq @ torch.linalg.inv(torch.where(alone[:, None, None], eye, aqq))
        g = 0.5 * (f.transpose(1, 2) @ f - eye)
        s2 = lam * torch.diagonal(g, dim1=1, dim2=2).sum(1)[:, None, None] * eye + mu2 * g
        stress = _sym(f @ s2 @ f.transpose(1, 2) / torch.linalg.det(f)[:, None, None])
        out["deformation"], out["stress"] = f, stress
    else:
        rot = torch.where((body > 0)[:, None, None], eye, _polar(torch.where((body > 0)[:, None, None], eye, apq)))
        q0, p0 = x0[j0] - x0[i0], x[j0] - x[i0]
        u = torch.einsum("nba,nb->na", rot[i0], p0) - q0
        dm = _sum(n, i0, u[:, :, None] * _grad(-q0, h)[:, None, :]) * (mass / rho0)[:, None, None]
        strain = torch.where((body > 0)[:, None], torch.zeros_like(_sym(dm)), _sym(dm))
        stress = mu2 * strain
        stress[:, :3] += lam * strain[:, :3].sum(1, keepdim=True)
        out["rotation"], out["strain"], out["stress"] = rot, strain, stress
    gw = _grad(x0[i0] - x0[j0], h) * (mass * mass / (rho0[i0] * rho0[j0]))[:, None]
    sig = full(stress)
    mv = lambda m, a: torch.einsum("nab,nb->na", m, a)  # noqa: E731
    own, other = mv(sig[i0], gw), mv(sig[j0], gw)
    other = torch.where((body[j0] > 0)[:, None], own, other)
    if not svk:
        own, other = mv(rot[i0], own), mv(rot[j0], other)
    fe = 0.5 * _sum(n, i0, own + other)
    r = (x[j] - x[i]).norm(dim=1)
    names = [k[0] for k in sc.entries]
    visc = _param(sc, "solid_viscosity" if "solid_viscosity" in names else "viscosity")
    lap = visc * mass / rho[j] * 45.0 / (PI * h ** 6) * (h - r).clamp_min(0)
    fv = _sum(n, i, (v[j] - v[i]) * lap[:, None])
    out.update({"density": rho, "force_elastic": fe, "force_viscous": fv, "force": fe + fv, "cutoff_force": fe + fv})
    return out


def _step(sc, x, v, f, moving):
    dt = _param(sc, "timestep")
    g = _f64(np.float32(sc.param("gravity")))
    a = torch.where(moving[:, None], f / _param(sc, "mass") + g, torch.zeros_like(f))
    v = torch.where(moving[:, None], v + dt * a, v)
    x = torch.where(moving[:, None], x + dt * v, x)
    if "wallbounds" in [k[0] for k in sc.entries]:
        w = _f64(np.float32(sc.param("wallbounds"))).reshape(3, 2)
        low, high = x < w[:, 0], x > w[:, 1]
        x = torch.where(low, 2 * w[:, 0] - x, torch.where(high, 2 * w[:, 1] - x, x))
        v = torch.where(low | high, -v, v)
    return x, v, a


def _advance(sc, x, v, x0=None):
    """One substep: (position, velocity, every other result)."""
    body = _f64(sc.init["body_number"]) if "body_number" in sc.init else torch.zeros_like(x[:, 0])
    h, mass = _param(sc, "smoothingradius"), _param(sc, "mass")
    if sc.material == "fluid":
        i, j = _pairs(x, h)
        rho = _density(x, i, j, h, mass)
        out = {"density": rho, "force": _fluid_force(sc, x, v, rho, i, j)}
    elif sc.material == "mixed":
        phase = _f64(sc.init["phase"])
        out = _solid(sc, x, v, x0, body, phase > 0, True)
        i, j = _pairs(x, h)
        elastic = torch.where((phase > 0)[:, None], out["force"], torch.zeros_like(x))
        out["force"] = elastic + _fluid_force(sc, x, v, out["density"], i, j, phase)
    else:
        out = _solid(sc, x, v, x0, body, torch.ones_like(body) > 0, sc.material == "svk")
    x, v, out["acceleration"] = _step(sc, x, v, out["force"], body == 0)
    return x, v, out


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        res = []
        for sc in _batch_scenes(case, seed):
            x0 = x = _f64(sc.init["position"])
            v = torch.zeros_like(x)
            for _ in range(BATCH_STEPS):
                x, v, _o = _advance(sc, x, v, x0)
            res.append(x.cpu())
        return res
    sc, later = _scene(case, seed)
    x0 = _f64(sc.init["position"])
    x = _f64(later["position"]) if "position" in later else x0
    v = _f64(later.get("velocity", sc.init.get("velocity", np.zeros((sc.n, 3), np.float32))))
    for _ in range(case.get("steps", 1)):
        x, v, out = _advance(sc, x, v, x0)
    if kind == "bar":
        on = sc.init["plane_constraints_particles"]
        last = float(np.float32(float(sc.init["position"][:, 0].max()) + 1e-4))
        for bit, at in ((1, float(np.float32(-1e-4))), (2, last)):
            m = torch.from_numpy((on & bit) > 0).to(x.device)
            x[m, 0], v[m, 0] = at, 0.0
        return dict(out, position=x, velocity=v)
    res = {name: out.get(name) for name in FIELDS[kind]}
    res["position"], res["velocity"] = x, v
    if kind == "mixed":
        # the ball moves as one body; only the solid phase has solid results
        res["position"] = res["velocity"] = res["acceleration"] = None
        for name in ("deformation", "stress", "force_elastic", "force_viscous", "cutoff_force"):
            res[name] = None
    return res
