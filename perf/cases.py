"""Workloads of the particle framework as its users run them, for timing.

A case is one call pattern of a program that uses the package: a frame (state
in from pinned host memory, some steps, state out), a pressure pre-solve, a
surface extraction, a training run of the warm-start network, a cell sort.
`listed()` names the standing set, `draw()` gives further cases of the same
ranges, `prepare()` builds what the program holds before the call, `run()`
makes the call, `exact()` gives the same outputs in 64-bit torch where they
have such a value.
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

import psb_project_b200 as psb

WARM = {"zero": psb.WARM_ZERO, "previous": psb.WARM_PREVIOUS, "learned": psb.WARM_LEARNED}


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # sorting one small cell population without allocating: the shortest call the library has
        dict(name="sort_5k", kind="sort", n=5000, bits=16),
        # the 16,384-particle WCSPH dam break, a frame of 8 steps: what an interactive front end runs
        dict(name="wcsph_16k", kind="wcsph", profile="config", nx=32, ny=32, nz=16, spacing=0.01, fx=3.125, fy=1.5625,
             fz=3.125, dt=5e-4, mass=1e-3, steps=8),
        # the 4,096-sphere DEM block of the coupled configuration, a frame of 16 steps
        dict(name="dem_4k", kind="dem", nx=16, ny=16, nz=16, steps=16),
        # the reference's own PCISPH (three fixed corrections, FP64 array-of-structures arrays), an odd size
        dict(name="ref_pci_100k", kind="ref", method="pcisph", nx=57, ny=41, nz=43, steps=3),
        # coupled fluid and spheres, 262,144 + 4,096, the boundary set handed over every step
        dict(name="coupled_262k", kind="coupled", nx=64, ny=64, nz=64, dem=16, steps=1),
        # pressure pre-solve before a run: the corrector's passes alone, ragged sizes
        dict(name="presolve_290k", kind="presolve", nx=67, ny=61, nz=71, spacing=0.01, fx=2.0, fy=1.5, fz=1.5, dt=1e-3,
             iters=32),
        # the 1,048,576-particle headline dam break, learned start, each step one graph launch
        dict(name="pci_1m", kind="pci", nx=128, ny=128, nz=64, spacing=0.005, fx=6.25, fy=3.125, fz=3.125, dt=5e-4,
             eta=0.01, warm="learned", graph=True, obstacle=0.0, steps=4),
        # a mid-size dam break stepped kernel by kernel from p = 0, ragged
        dict(name="pci_97k", kind="pci", nx=47, ny=53, nz=39, spacing=0.01, fx=2.5, fy=1.7, fz=1.3, dt=5e-4, eta=0.01,
             warm="zero", graph=False, obstacle=0.0, steps=4),
        # the largest scene: 4,194,304 particles around a sphere of boundary particles, eta 0.5 %
        dict(name="pci_4m_obstacle", kind="pci", nx=256, ny=128, nz=128, spacing=0.004, fx=2.93, fy=2.93, fz=1.953,
             dt=5e-4, eta=0.005, warm="previous", graph=True, obstacle=0.2, steps=2),
        # 64 independent scenes of 4k to 131k particles in one context
        dict(name="batch_64", kind="batch", scenes=64, lo=4096, hi=131072, warm="previous", steps=2),
        # colour field and marching cubes on 128^3 nodes over a 262,144-particle scene
        dict(name="surface_128", kind="surface", nx=64, ny=64, nz=64, nodes=128),
        # 64 Adam steps of the warm-start network on recorded rows
        dict(name="mlp_train_64", kind="mlp", nx=32, ny=32, nz=32, arch=0, batch=65536, iters=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _block(rng, lo, hi):
    """Edge counts of a lattice block of about lo..hi particles, its edges within a factor of 2."""
    n = _log(rng, lo, hi)
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    e = (n / (a * b)) ** (1 / 3)
    return dict(nx=max(4, round(e * a)), ny=max(4, round(e * b)), nz=max(4, round(e)))


def _box(rng):
    return dict(fx=round(rng.uniform(1.6, 4.0), 3), fy=round(rng.uniform(1.4, 2.5), 3), fz=round(rng.uniform(1.2, 2.5), 3))


def draw(rng):
    kind = rng.choice(["sort", "wcsph", "dem", "ref", "coupled", "presolve", "pci", "pci", "batch", "surface", "mlp"])
    if kind == "sort":
        return dict(kind=kind, n=_log(rng, 200, 262144), bits=rng.randint(6, 32))
    if kind == "wcsph":
        return dict(kind=kind, profile=rng.choice(["config", "ref"]), **_block(rng, 1000, 120000), spacing=0.01,
                    **_box(rng), dt=5e-4, mass=1e-3, steps=rng.randint(4, 12))
    if kind == "dem":
        return dict(kind=kind, **_block(rng, 400, 30000), steps=rng.randint(8, 24))
    if kind == "ref":
        return dict(kind=kind, method=rng.choice(["pcisph", "pcisph", "wcsph"]), **_block(rng, 4000, 400000),
                    steps=rng.randint(1, 4))
    if kind == "coupled":
        return dict(kind=kind, **_block(rng, 12000, 200000), dem=rng.randint(5, 14), steps=rng.randint(1, 2))
    if kind == "presolve":
        return dict(kind=kind, **_block(rng, 8000, 500000), spacing=0.01, **_box(rng), dt=1e-3,
                    iters=rng.randint(16, 64))
    if kind == "pci":
        return dict(kind=kind, **_block(rng, 6000, 1500000), spacing=rng.choice([0.004, 0.005, 0.01]), **_box(rng),
                    dt=5e-4, eta=rng.choice([0.01, 0.005]), warm=rng.choice(["zero", "previous", "learned"]),
                    graph=rng.random() < 0.7, obstacle=rng.choice([0.0, 0.0, 0.15]), steps=rng.randint(1, 4))
    if kind == "batch":
        lo = _log(rng, 1000, 8000)
        return dict(kind=kind, scenes=_log(rng, 2, 64), lo=lo, hi=lo * rng.randint(2, 10),
                    warm=rng.choice(["zero", "previous", "learned"]), steps=rng.randint(1, 3))
    if kind == "surface":
        return dict(kind=kind, **_block(rng, 12000, 400000), nodes=rng.randint(40, 160))
    return dict(kind=kind, nx=rng.randint(18, 36), ny=rng.randint(18, 36), nz=rng.randint(18, 36), arch=rng.randint(0, 1),
                batch=_log(rng, 2000, 131072), iters=rng.randint(16, 96))


# ---- scenes and their states ----------------------------------------------------

def _pinned(shape, dtype=torch.float32):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _fluid_scene(c, seed):
    n, s = (c["nx"], c["ny"], c["nz"]), c.get("spacing", 0.01)
    box = tuple(round(m * s * c[f], 3) for m, f in zip(n, ("fx", "fy", "fz")))
    kind = c["kind"]
    profile = psb.PROFILE_REF if c.get("profile") == "ref" else psb.PROFILE_CONFIG
    sc = psb.dam_break(n, s, box, 2 * s, method=psb.WCSPH if kind == "wcsph" else psb.PCISPH, profile=profile,
                       dt=c["dt"], mass=c.get("mass"), eta=c.get("eta", 0.01), seed=seed)
    return sc.replace(warm_start=WARM[c.get("warm", "zero")])


def _ref_scene(c, seed):
    n, s = (c["nx"], c["ny"], c["nz"]), 0.01
    sc = psb.ref_scene(n, s, tuple(round(m * s * f, 3) for m, f in zip(n, (2.0, 1.5, 1.5))), 2 * s,
                       method=psb.WCSPH if c["method"] == "wcsph" else psb.PCISPH, seed=seed)
    return sc.replace(spacing=s)


def _coupled_scenes(c, seed):
    if (c["nx"], c["ny"], c["nz"], c["dem"]) == (64, 64, 64, 16):
        return psb.c1_scenes(seed=seed)
    s, h = 0.01, 0.02
    n, m = (c["nx"], c["ny"], c["nz"]), c["dem"]
    top = n[1] * s
    box = (max(2 * n[0] * s, 0.021 * m + 0.2), top + 0.021 * m + 0.1, max(1.3 * n[2] * s, 0.021 * m + 0.2))
    box = tuple(round(b, 3) for b in box)
    fluid = psb.dam_break(n, s, box, h, dt=1e-3, mass=1e-3, seed=seed)
    spheres = psb.dem_block((m, m, m), 0.021, (0.1, top + 0.02, 0.1), box, 0.01, dt=1e-3, seed=seed + 100)
    return fluid, spheres


def _batch_scenes(c, seed):
    """The boxes and sizes of the configured batch; the seed moves the particles."""
    scenes = psb.batch_scenes(c["scenes"], n_range=(c["lo"], c["hi"]), warm_start=WARM[c["warm"]])
    return [s.replace(blocks=[dataclasses.replace(b, seed=seed * 1000 + k) for b in s.blocks])
            for k, s in enumerate(scenes)]


def _motion(pos, extent, g, seed, speed=0.5):
    """Velocities and pressures of a block in motion: one roll in the xy plane
    that is tangent to the block's faces, a little particle noise, and the
    hydrostatic pressure of the column above."""
    rng = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.as_tensor(pos, device="cuda")
    a, b = extent[0], extent[1]
    u, w = math.pi * x[:, 0] / a, math.pi * x[:, 1] / b
    v = torch.empty_like(x)
    v[:, 0] = speed * torch.sin(u) * torch.cos(w)
    v[:, 1] = -speed * (b / a) * torch.cos(u) * torch.sin(w)
    v[:, 2] = 0.1 * speed * torch.sin(u) * torch.sin(w)
    v += 0.005 * speed * torch.randn(x.shape, generator=rng, device="cuda")
    p = 1000.0 * g * (b - x[:, 1]).clamp(min=0)
    p *= 1 + 0.05 * torch.randn(p.shape, generator=rng, device="cuda")
    vel, pres = _pinned(tuple(v.shape)), _pinned(tuple(p.shape))
    vel[:] = v.cpu().numpy()
    pres[:] = p.clamp(min=0).cpu().numpy()
    return vel, pres


def _extent(sc):
    b = sc.blocks[0]
    return [m * b.spacing for m in b.nxyz]


def _positions(sc):
    pos = psb.scene_positions(sc)
    out = _pinned(pos.shape)
    out[:] = pos
    return out


def _out(n):
    return {"pos": _pinned((n, 3)), "vel": _pinned((n, 3)), "vel_half": _pinned((n, 3)), "density": _pinned(n),
            "pressure": _pinned(n)}


def _weights(arch, seed):
    """A network that leans on the carried pressure (input 3), as a trained one
    does: silu(x) - silu(-x) = relu(x) - relu(-x) = x carries it through both
    layers; the other units are small and random."""
    w = psb.mlp_init_weights(seed, arch) * np.float32(0.05)
    W1, _, W2, _, W3, _ = psb.mlp_unpack(w)
    W1[:2] = 0
    W1[0, 3], W1[1, 3] = 1, -1
    W2[:2] = 0
    W2[0, 0], W2[0, 1], W2[1, 0], W2[1, 1] = 1, -1, -1, 1
    W3[0], W3[1] = 0.95, -0.95
    return w


def _obstacle(c, sc):
    """A sphere shell of boundary particles on the floor, clear of the block."""
    ext, box, s = _extent(sc), sc.box_max, sc.blocks[0].spacing
    r = min(c["obstacle"], 0.2 * min(box[1], box[2]), 0.35 * (box[0] - ext[0]))
    return psb.sphere_shell((ext[0] + r + 1.5 * s, r, 0.5 * box[2]), r, s)


# ---- prepare ----------------------------------------------------------------------

def prepare(case, seed):
    c = case
    kind = c["kind"]
    if kind == "sort":
        rng = torch.Generator(device="cuda").manual_seed(seed)
        top = 1 << c["bits"]
        keys = torch.randint(0, top, (c["n"],), generator=rng, device="cuda", dtype=torch.int64)
        keys = torch.where(keys >= 1 << 31, keys - (1 << 32), keys).to(torch.int32)
        vals = torch.randperm(c["n"], generator=rng, device="cuda").to(torch.int32)
        return {"case": c, "keys": keys, "vals": vals, "keys_out": torch.empty_like(keys),
                "vals_out": torch.empty_like(vals)}
    if kind == "coupled":
        fs, ds = _coupled_scenes(c, seed)
        fluid, spheres = psb.Simulation(fs), psb.Simulation(ds)
        pos, dpos = _positions(fs), _positions(ds)
        vel, pres = _motion(pos, _extent(fs), 9.81, seed)
        dvel = _pinned(dpos.shape)
        dvel[:] = np.random.default_rng(seed).normal(0, 0.05, dpos.shape) + np.float32([0, -0.5, 0])
        return {"case": c, "fluid": fluid, "spheres": spheres, "pair": psb.FluidDemCoupling(fluid, spheres),
                "in": (pos, vel, vel, pres), "dem_in": (dpos, dvel, dvel), "out": _out(fs.n), "dem_out": _out(ds.n)}
    if kind == "batch":
        scenes = _batch_scenes(c, seed)
        sim = psb.BatchSimulation(scenes)
        pos = np.concatenate([psb.scene_positions(s) for s in scenes])
        vel, pres = _pinned(pos.shape), _pinned(len(pos))
        for s, a, b in zip(scenes, sim.first[:-1], sim.first[1:]):
            vel[a:b], pres[a:b] = _motion(pos[a:b], _extent(s), 9.81, seed + int(a))
        if c["warm"] == "learned":
            sim.mlp_set_weights(_weights(0, seed))
        sim.set_graph(True)
        pin = _pinned(pos.shape)
        pin[:] = pos
        return {"case": c, "sim": sim, "in": (pin, vel, vel, pres), "out": _out(len(pos))}
    if kind == "dem":
        sc = _dem_scene(c, seed)
        sim = psb.Simulation(sc)
        pos = _positions(sc)
        vel = _pinned(pos.shape)
        vel[:] = np.random.default_rng(seed).normal(0, 0.2, pos.shape)
        return {"case": c, "sim": sim, "in": (pos, vel, vel, None), "out": _out(sc.n)}
    if kind == "ref":
        sc = _ref_scene(c, seed)
        sim = psb.Simulation(sc)
        pos = _positions(sc)
        vel, _ = _motion(pos, _extent(sc), 9.81, seed)
        dev = [torch.as_tensor(a, device="cuda").double() for a in (pos, vel)]
        return {"case": c, "sim": sim, "pos": dev[0], "vel": dev[1]}
    if kind == "mlp":
        sc = psb.dam_break((c["nx"], c["ny"], c["nz"]), 0.01, (1.0, 0.6, 0.6), 0.02, dt=5e-4, seed=seed)
        sim = psb.Simulation(sc)
        pos = _positions(sc)
        vel, pres = _motion(pos, _extent(sc), 9.81, seed)
        sim.upload(pos, vel, vel, pres)
        sim.mlp_set_arch(c["arch"])
        sim.mlp_collect(2, 1 << 19)
        sim.step(10)
        return {"case": c, "sim": sim, "w": psb.mlp_init_weights(seed, c["arch"])}
    if kind == "surface":
        n, s = (c["nx"], c["ny"], c["nz"]), 0.01
        box = tuple(round(m * s * f, 3) for m, f in zip(n, (1.6, 1.4, 1.3)))
        sc = psb.dam_break(n, s, box, 2 * s, dt=5e-4, seed=seed)
        sim = psb.Simulation(sc)
        pos = _positions(sc)
        vel, pres = _motion(pos, _extent(sc), 9.81, seed)
        sim.upload(pos, vel, vel, pres)
        sim.step(1)
        k = c["nodes"]
        lo, hi = [-2 * s] * 3, [1.1 * e + 2 * s for e in _extent(sc)]
        grid = psb.iso_grid(lo, [(b - a) / (k - 1) for a, b in zip(lo, hi)], (k, k, k))
        vert, tri = _pinned((12 * k * k, 3)), _pinned((24 * k * k, 3), torch.int32)
        vert[:], tri[:] = 0, 0
        return {"case": c, "sim": sim, "grid": grid, "vert": vert, "tri": tri}
    sc = _fluid_scene(c, seed)         # wcsph, presolve, pci
    sim = psb.Simulation(sc)
    pos = _positions(sc)
    vel, pres = _motion(pos, _extent(sc), 9.81, seed)
    if kind == "pci":
        if c["obstacle"]:
            sim.set_boundary(_obstacle(c, sc))
        if c["warm"] == "learned":
            sim.mlp_set_weights(_weights(0, seed))
        if c["graph"]:
            sim.set_graph(True)
    return {"case": c, "sim": sim, "in": (pos, vel, vel, pres), "out": _out(sc.n)}


def _dem_scene(c, seed):
    n = (c["nx"], c["ny"], c["nz"])
    box = tuple(round(0.0195 * m + e, 3) for m, e in zip(n, (0.5, 0.3, 0.3)))
    # spheres of radius 0.01 at 0.0195: neighbours just in contact, as in a settled bed
    return psb.dem_block(n, 0.0195, (0.0, 0.0, 0.0), box, 0.01, dt=1e-4, seed=seed)


# ---- run ----------------------------------------------------------------------------

def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "sort":
        rc = psb.lib().psb_sort_cells_noalloc(state["keys"].data_ptr(), state["vals"].data_ptr(),
                                              state["keys_out"].data_ptr(), state["vals_out"].data_ptr(), c["n"],
                                              c["bits"], torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError("psb_sort_cells_noalloc: %d" % rc)
        return state["keys_out"], state["vals_out"]
    if kind == "coupled":
        fluid, spheres = state["fluid"], state["spheres"]
        fluid.upload(*state["in"])
        spheres.upload(*state["dem_in"])
        state["pair"].step(c["steps"])
        return fluid.download(state["out"]), spheres.download(state["dem_out"]), state["pair"].last_force
    sim = state["sim"]
    if kind == "ref":
        sim.upload_aos_f64(state["pos"].data_ptr(), state["vel"].data_ptr(), state["vel"].data_ptr(), on_device=True)
        sim.n = c["nx"] * c["ny"] * c["nz"]
        sim.step(c["steps"])
        return sim.download_aos_f64()
    if kind == "mlp":
        sim.mlp_set_weights(state["w"])
        loss = sim.mlp_train(c["iters"], c["batch"], 3e-3, seed=1)
        return sim.mlp_get_weights(), loss
    if kind == "surface":
        nv, nt = sim.extract_surface_into(state["grid"], 0.5, state["vert"], state["tri"])
        return state["vert"], state["tri"], nv, nt
    sim.upload(*state["in"])
    if kind == "presolve":
        sim.presolve(c["iters"])
        return sim.download({"density": state["out"]["density"], "pressure": state["out"]["pressure"]})
    sim.step(c["steps"])
    return sim.download(state["out"])


# ---- work ---------------------------------------------------------------------------

# Pairs per particle of a filled neighbourhood (h = 2 spacings, self
# included), and the operations of one pair in a density sum, in the set-up
# forces, in a pressure-force sum and in the velocity smoothing.
_PAIRS, _DENSITY, _FORCES, _PRESSURE, _XSPH = 33, 16, 40, 26, 20


def work(case):
    """State in and out once per step; the pair sums no formulation avoids,
    with the smallest number of corrections the method allows."""
    c = case
    kind = c["kind"]
    if kind == "sort":
        return {"bytes": 16 * c["n"], "flops": 0}
    if kind == "mlp":
        p = 64 * (6 + c["arch"]) + 64 * 64 + 64
        return {"bytes": c["iters"] * c["batch"] * 36, "flops": c["iters"] * c["batch"] * 6 * p}
    if kind == "batch":
        mean = (c["hi"] - c["lo"]) / math.log(c["hi"] / c["lo"])
        n = c["scenes"] * mean
    else:
        n = c["nx"] * c["ny"] * c["nz"]
    if kind == "surface":
        nodes = c["nodes"] ** 3
        return {"bytes": 24 * n + 8 * nodes + 36 * 6 * c["nodes"] ** 2,
                "flops": n * (_PAIRS * _DENSITY + nodes / n * 33 * 12)}
    if kind == "dem":
        return {"bytes": c["steps"] * n * 64, "flops": c["steps"] * n * 7 * 30}
    if kind == "wcsph" or (kind == "ref" and c["method"] == "wcsph"):
        return {"bytes": c["steps"] * n * 84, "flops": c["steps"] * n * _PAIRS * (_DENSITY + _FORCES + _PRESSURE)}
    if kind == "presolve":
        return {"bytes": n * 48, "flops": n * _PAIRS * (_DENSITY + _FORCES + c["iters"] * (_DENSITY + _PRESSURE))}
    sums = _DENSITY + _FORCES + 3 * (_DENSITY + _PRESSURE) + (0 if kind == "ref" else _DENSITY + _XSPH)
    return {"bytes": c["steps"] * n * 84, "flops": c["steps"] * n * _PAIRS * sums}


# ---- the same in 64 bits -----------------------------------------------------------------

def _pairs(x, h):
    """(i, j) of all pairs with |x_i - x_j| <= h, self included."""
    lo = x.min(0).values - h
    cell = ((x - lo) / h).floor().long()
    dims = (cell.max(0).values + 2).tolist()
    key = cell[:, 0] + dims[0] * (cell[:, 1] + dims[1] * cell[:, 2])
    order = torch.argsort(key)
    skey = key[order]
    ncell = dims[0] * dims[1] * dims[2]
    count = torch.bincount(skey, minlength=ncell)
    start = torch.cumsum(count, 0) - count
    most = int(count.max())
    ii, jj = [], []
    idx = torch.arange(len(x), device=x.device)
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                k = key + dx + dims[0] * (dy + dims[1] * dz)
                for m in range(most):
                    i = idx[count[k] > m]
                    if not len(i):
                        break
                    j = order[start[k[i]] + m]
                    near = (x[i] - x[j]).square().sum(1) <= h * h
                    ii.append(i[near])
                    jj.append(j[near])
    return torch.cat(ii), torch.cat(jj)


class _Exact:
    """SPH and DEM steps of one scene in 64-bit torch."""

    def __init__(self, sc, pos, vel, vap, p=None):
        t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device="cuda")  # noqa: E731
        self.sc, self.x, self.v, self.vap = sc, t(pos), t(vel), t(vap)
        n = len(self.x)
        self.p = t(p) if p is not None else torch.zeros(n, dtype=torch.float64, device="cuda")
        self.rho = torch.zeros_like(self.p)
        f = np.float32
        self.ref = sc.profile == psb.PROFILE_REF
        self.dt, self.r = float(f(sc.dt)), float(f(sc.particle_radius))
        self.b0, self.b1 = [[float(f(b)) for b in v] for v in (sc.box_min, sc.box_max)]
        h, m = sc.h, sc.mass
        self.g = [float(f(a)) for a in ((0, -9.81, 0) if self.ref and sc.method == psb.PCISPH else sc.gravity)]
        self.k_rho = 315 * m / (64 * math.pi * h ** 3)
        self.G = 45 / (math.pi * h ** 4)
        self.k_grad = m * self.G
        self.k_visc = sc.mu * m * 45 / (math.pi * h ** 5)
        self.k_surf = 945 * m / (32 * math.pi * h ** 5)
        self.sigma = 0.0728 if sc.method == psb.PCISPH else sc.sigma
        beta = 2 * (m * self.dt / sc.rho0) ** 2
        self.k_press = 1 / (beta * self.G ** 2)
        s, R = sc.spacing, int(math.ceil(h / sc.spacing))
        w2 = 0.0
        for i in range(-R, R + 1):
            for j in range(-R, R + 1):
                for k in range(-R, R + 1):
                    d = s * math.sqrt(i * i + j * j + k * k)
                    if 0 < d < h:
                        w2 += (self.G * (1 - d / h) ** 2) ** 2
        self.k_delta = 1 / (beta * w2) if w2 else 0.0     # the gradients of a full lattice cancel

    def add(self, i, w):
        out = torch.zeros((len(self.x),) + tuple(w.shape[1:]), dtype=torch.float64, device="cuda")
        return out.index_add_(0, i, w)

    def build(self):
        self.i, self.j = _pairs(self.x, self.sc.h)

    def walls(self, x):
        """Ghost pairs of the box faces near x_i: (pair index, offset, hydrostatic term)."""
        h = self.sc.h
        near = []
        for a in range(3):
            lower = x[:, a] - self.b0[a] < h
            upper = ~lower & (self.b1[a] - x[:, a] < h)
            near.append((lower, upper))
        for mask in range(1, 8):
            ok = torch.ones(len(x), dtype=torch.bool, device="cuda")
            for a in range(3):
                if mask >> a & 1:
                    ok &= near[a][0] | near[a][1]
            at = torch.nonzero(ok[self.i])[:, 0]
            if not len(at):
                continue
            i, j = self.i[at], self.j[at]
            r = x[i] - x[j]
            dp = torch.zeros(len(at), dtype=torch.float64, device="cuda")
            keep = torch.ones(len(at), dtype=torch.bool, device="cuda")
            for a in range(3):
                if not mask >> a & 1:
                    continue
                lower = near[a][0][i]
                nrm = torch.where(lower, 1.0, -1.0).double()
                plane = torch.where(lower, self.b0[a], self.b1[a]).double()
                dj = (nrm * (x[j, a] - plane)).clamp(min=0)
                di = (nrm * (x[i, a] - plane)).clamp(min=0)
                keep &= dj < h
                r[:, a] = nrm * (di + dj)
                dp += self.sc.rho0 * (-self.g[a] * nrm) * 2 * dj
            yield i[keep], j[keep], r[keep], dp[keep]

    def density(self, x):
        h2 = self.sc.h ** 2
        q = (x[self.i] - x[self.j]).square().sum(1) / h2
        w = (1 - q) if self.ref else (1 - q).clamp(min=0)
        rho = self.add(self.i, w ** 3)
        if not self.ref:
            for i, _, r, _ in self.walls(x):
                rho += self.add(i, (1 - r.square().sum(1) / h2).clamp(min=0) ** 3)
        return self.k_rho * rho

    def spiky(self, r):
        """r^ (1 - |r|/h)^2 inside the support, 0 at r = 0."""
        d = r.square().sum(1).sqrt()
        om = 1 - d / self.sc.h
        s = torch.where(d > 0, om ** 2 / d.clamp(min=1e-300), torch.zeros_like(d))
        return s if self.ref else torch.where(om > 0, s, torch.zeros_like(s))

    def pressure_accel(self, x, p, rho):
        pv = p / rho ** 2 if self.ref else p / self.sc.rho0 ** 2
        r = x[self.i] - x[self.j]
        a = self.add(self.i, ((pv[self.i] + pv[self.j]) * self.spiky(r))[:, None] * r)
        if not self.ref:
            for i, j, r, dp in self.walls(x):
                a += self.add(i, ((pv[i] + (p[j] + dp) / self.sc.rho0 ** 2) * self.spiky(r))[:, None] * r)
        return self.k_grad * a

    def force(self, rho):
        """Viscosity, surface tension (reference) and gravity force density at x."""
        i, j = self.i, self.j
        r = self.x[i] - self.x[j]
        d2 = r.square().sum(1)
        on = d2 > 0
        u = d2.sqrt() / self.sc.h
        near = on if self.ref else on & (u < 1)
        sv = torch.where(near, (1 - u) / rho[j], torch.zeros_like(u))
        f = self.k_visc * self.add(i, (self.v[j] - self.v[i]) * sv[:, None])
        if self.ref:
            t = torch.where(on, 1 - u * u, torch.zeros_like(u))
            nrm = -self.k_surf * self.add(i, r * (t * t / rho[j])[:, None])
            fs = -self.k_surf * self.add(i, torch.where(on, t * (3 - 7 * u * u) / rho[j], torch.zeros_like(u)))
            ln = nrm.square().sum(1).sqrt()
            c = torch.where(ln >= self.sc.l, -fs * self.sigma / ln.clamp(min=1e-300), torch.zeros_like(ln))
            f += c[:, None] * nrm
        return f + rho[:, None] * torch.tensor(self.g, dtype=torch.float64, device="cuda")

    def wall_accel(self):
        a = torch.zeros_like(self.x)
        if not self.ref:
            k, c = float(np.float32(self.sc.wall_k)), float(np.float32(self.sc.wall_c))
            for d in range(3):
                lo, hi = self.b0[d] - self.x[:, d], self.b1[d] - self.x[:, d]
                a[:, d] += torch.where(lo > 0, k * lo - c * self.vap[:, d], torch.zeros_like(lo))
                a[:, d] += torch.where(hi < 0, k * hi - c * self.vap[:, d], torch.zeros_like(hi))
        return a

    def project(self, x, v):
        n = torch.zeros_like(x)
        y = x.clone()
        for d in range(3):
            hi, lo = float(np.float32(self.b1[d]) - np.float32(self.r)), float(np.float32(self.b0[d]) + np.float32(self.r))
            for at, b, s in ((x[:, d] >= hi, hi, -1.0), (x[:, d] <= lo, lo, 1.0)):
                y[at, d] = b
                n[at, d] = s
        ln = n.square().sum(1, keepdim=True).sqrt()
        n = n / ln.clamp(min=1e-300)
        return y, v - (v * n).sum(1, keepdim=True) * n

    def wcsph(self):
        self.build()
        sc = self.sc
        self.rho = self.density(self.x)
        if self.ref:
            self.p = sc.k * (self.rho - sc.rho0)
        else:
            self.p = sc.k * sc.rho0 / 7 * ((self.rho / sc.rho0) ** 7 - 1)
        a = self.force(self.rho) / self.rho[:, None] + self.pressure_accel(self.x, self.p, self.rho) + self.wall_accel()
        v = self.vap + a * self.dt
        x = self.x + v * self.dt
        if self.ref:
            x, v = self.project(x, v)
        self.v, self.vap, self.x = (self.vap + v) / 2, v, x

    def begin(self, warm):
        self.build()
        rho = self.density(self.x)
        if not warm:
            self.p = torch.zeros_like(self.p)
        self.f, self.aw = self.force(rho), self.wall_accel()
        a = self.f / rho[:, None] + self.aw
        if warm:
            a = a + self.pressure_accel(self.x, self.p, rho)
        self.vs = self.vap + a * self.dt
        self.xs = self.x + self.vs * self.dt
        self.rho = rho

    def candidate(self):
        rho = self.density(self.xs)
        d = rho - self.sc.rho0
        if self.ref:
            r = self.xs[self.i] - self.xs[self.j]
            s = self.spiky(r)
            t1, t2 = self.add(self.i, s[:, None] * r), self.add(self.i, s * s * r.square().sum(1))
            den = t1.square().sum(1) + t2
            on = (d > 0) & (t2 > 0)
            p = torch.where(on, self.p + self.k_press * d / torch.where(on, den, torch.ones_like(den)), self.p)
        else:
            p = (self.p + self.k_delta * d).clamp(min=0)
        return rho, p, float(d.max()) / self.sc.rho0

    def correct(self, rho, p):
        a = self.f / rho[:, None] + self.pressure_accel(self.xs if self.ref else self.x, p, rho) + self.aw
        self.vs = self.vap + a * self.dt
        self.xs = self.x + self.vs * self.dt
        self.rho, self.p = rho, p

    def pcisph(self):
        sc = self.sc
        self.begin(not self.ref and sc.warm_start != psb.WARM_ZERO)
        for k in range(3 if self.ref else sc.max_iters):
            rho, p, err = self.candidate()
            if not self.ref and k >= sc.min_iters and err <= sc.eta:
                break
            self.correct(rho, p)
        self.rho = rho
        if sc.xsph and not self.ref:
            q = ((self.xs[self.i] - self.xs[self.j]).square().sum(1) / sc.h ** 2)
            w = (1 - q).clamp(min=0) ** 3 * (sc.xsph * self.k_rho / sc.rho0)
            self.vs = self.vs + self.add(self.i, w[:, None] * (self.vs[self.j] - self.vs[self.i]))
        x, v = self.project(self.xs, self.vs)
        self.v, self.vap, self.x = (self.vap + v) / 2, v, x

    def presolve(self, iters):
        self.begin(True)
        for _ in range(iters):
            rho, p, _ = self.candidate()
            self.correct(rho, p)

    def dem(self):
        sc = self.sc
        self.build()
        k, c = float(np.float32(sc.dem_spring)), float(np.float32(sc.dem_damping))
        R = float(np.float32(2 * sc.particle_radius))
        r = self.x[self.j] - self.x[self.i]
        d = r.square().sum(1).sqrt()
        on = (d > 0) & (d < R)
        i, j, r, d = self.i[on], self.j[on], r[on], d[on]
        nrm = r / d[:, None]
        s = -k * (R - d) + c * ((self.v[j] - self.v[i]) * nrm).sum(1)
        f = self.add(i, s[:, None] * nrm) + sc.mass * torch.tensor(self.g, dtype=torch.float64, device="cuda")
        v = self.v + f / sc.mass * self.dt
        self.x, self.v = self.project(self.x + v * self.dt, v)
        self.vap = self.v

    def state(self, names=("pos", "vel", "vel_half", "density", "pressure")):
        got = {"pos": self.x, "vel": self.v, "vel_half": self.vap, "density": self.rho, "pressure": self.p}
        return {k: got[k].cpu().numpy() for k in names}


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "sort":
        s = prepare(c, seed)
        keys, at = torch.sort(s["keys"].long() & 0xFFFFFFFF, stable=True)
        return torch.where(keys >= 1 << 31, keys - (1 << 32), keys).to(torch.int32), s["vals"][at]
    # a trained BF16 network, a welded mesh and the coupled pair have no value of their own in 64 bits
    if kind in ("mlp", "surface", "coupled") or c.get("warm") == "learned" or c.get("obstacle"):
        return None
    if kind == "batch":
        if c["scenes"] * c["hi"] > 400000:
            return None
        s = prepare(c, seed)
        parts, first = [], s["sim"].first
        for sc, a, b in zip(_batch_scenes(c, seed), first[:-1], first[1:]):
            e = _Exact(sc, *[v[a:b] for v in s["in"]])
            for _ in range(c["steps"]):
                e.pcisph()
            parts.append(e.state())
        return {k: np.concatenate([p[k] for p in parts]) for k in parts[0]}
    if c["nx"] * c["ny"] * c["nz"] > 400000:
        return None
    s = prepare(c, seed)
    if kind == "ref":
        pos, vel = s["pos"].cpu().numpy(), s["vel"].cpu().numpy()
        e = _Exact(_ref_scene(c, seed), pos, vel, vel)
    elif kind == "dem":
        e = _Exact(_dem_scene(c, seed), *s["in"])
    else:
        e = _Exact(_fluid_scene(c, seed), *s["in"])
    if kind == "presolve":
        e.presolve(c["iters"])
        return e.state(("density", "pressure"))
    step = {"dem": e.dem, "wcsph": e.wcsph}.get(kind, e.wcsph if c.get("method") == "wcsph" else e.pcisph)
    for _ in range(c["steps"]):
        step()
    return e.state(("pos", "vel", "vel_half") if kind == "ref" else ("pos", "vel", "vel_half", "density", "pressure"))
