"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is a dict of plain values; `prepare` makes what a user's program has in hand before the call
(a configured simulation, its start state, pinned output arrays), `run` is one pass through the
public entry points, `exact` the same result in plain torch at 64 bits where it has one.

Kinds:
- "bed": the XPBD step of spheres in a closed box, in a packed bed (a touching lattice with jitter;
  `settled`: the saved settled 4,096-sphere bed of the settling configuration). A pass starts the
  simulation again from its state (as a parameter study does), runs one outer step (10 substeps of
  1e-5 s) and reads the state back.
- "periodic": polydisperse spheres in a box periodic in x and y on a floor: one outer step of a
  running simulation, then the state read back.
- "drums": independent rotating drums stepped together (the batched form): as "periodic".
- "shells": hollow cylinders with a point shell: as "bed", 8 substeps.
- "hertz": the explicit Hertz engine, polydisperse spheres in one SDF-wall box: one call of a running
  simulation, then the state read back.
- "calibration": forward and adjoint of the differentiable Hertz rollout, boxes of spheres.
- "xpbd_adjoint": forward and adjoint of the XPBD rollout on a packed bed.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "peclet-dem_b200"))

R0 = 1e-3  # grain radius, m
DENSITY = 2500.0
HZ = {"youngs": 1e7, "poisson": 0.3, "e": 0.6, "mu": 0.4}
THETA = (4e6, 0.6, 0.3)  # (E, e, mu) of the calibration rollouts


def listed():
    return [
        # a probe-sized column: the smallest calls, where launches and read-backs count
        {"name": "column_64_fp64", "kind": "bed", "n": 64, "precision": "fp64", "settled": False},
        # an ordinary bed with a ragged top layer, in the reference's own precision
        {"name": "bed_1021_fp32", "kind": "bed", "n": 1021, "precision": "fp32", "settled": False},
        # the settling configuration's bed at rest: the benchmark's headline
        {"name": "settled_4096_fp64", "kind": "bed", "n": 4096, "precision": "fp64", "settled": True},
        # a large packed bed: every solve loop runs its full sweeps over some 60,000 contacts
        {"name": "bed_20011_fp64", "kind": "bed", "n": 20011, "precision": "fp64", "settled": False},
        # the large polydisperse packing, periodic in x and y (ghost images, few sweeps)
        {"name": "periodic_262144_fp64", "kind": "periodic", "n": 262144, "precision": "fp64"},
        # a rotating-drum study: many uneven scenes in one simulation
        {"name": "drums_64_fp64", "kind": "drums", "scenes": 64, "nmin": 256, "nmax": 8192, "precision": "fp64"},
        {"name": "drums_256_mixed", "kind": "drums", "scenes": 256, "nmin": 256, "nmax": 4096, "precision": "mixed"},
        # non-spherical grains in line contact: some 80 shell-point contacts a body
        {"name": "shells_216_mixed", "kind": "shells", "n": 216, "points": 512, "precision": "mixed"},
        # the soft-sphere engine, a small calibration packing and the large one
        {"name": "hertz_2003_fp64", "kind": "hertz", "n": 2003, "substeps": 100, "precision": "fp64"},
        {"name": "hertz_262144_fp32", "kind": "hertz", "n": 262144, "substeps": 100, "precision": "fp32"},
        # gradients of (E, e, mu) and the start velocities over independent boxes
        {"name": "calibration_64x2048_fp64", "kind": "calibration", "scenes": 64, "nx": 8, "ny": 8, "nz": 32,
         "substeps": 200, "precision": "fp64"},
        # gradients through the XPBD substep on a packed bed
        {"name": "xpbd_adjoint_2197_fp64", "kind": "xpbd_adjoint", "n": 2197, "substeps": 10},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["bed", "bed", "bed", "periodic", "drums", "shells", "hertz", "calibration", "xpbd_adjoint"])
    prec = rng.choice(["fp64", "fp64", "fp32", "mixed"])
    if kind == "bed":
        return {"kind": kind, "n": log_int(27, 20000), "precision": prec, "settled": False}
    if kind == "periodic":
        return {"kind": kind, "n": log_int(1000, 262144), "precision": prec}
    if kind == "drums":
        return {"kind": kind, "scenes": log_int(3, 160), "nmin": rng.choice([64, 256]), "nmax": rng.choice([1024, 4096]),
                "precision": prec}
    if kind == "shells":
        return {"kind": kind, "n": log_int(20, 200), "points": rng.choice([131, 256, 512]), "precision": prec}
    if kind == "hertz":
        return {"kind": kind, "n": log_int(500, 250000), "substeps": rng.choice([10, 37, 100]),
                "precision": rng.choice(["fp64", "fp32"])}
    if kind == "calibration":
        return {"kind": kind, "scenes": log_int(1, 48), "nx": rng.randint(3, 8), "ny": rng.randint(3, 8),
                "nz": rng.randint(5, 32), "substeps": rng.choice([64, 120, 200]), "precision": rng.choice(["fp64", "fp32"])}
    return {"kind": kind, "n": log_int(27, 2100), "substeps": rng.randint(3, 10)}


# ---- inputs ---------------------------------------------------------------------------------------
def _inertia(r, density=DENSITY):
    m = density * 4.0 / 3.0 * np.pi * r ** 3
    return m, 0.4 * m * r * r


def _lattice(n, nx, ny, pitch, rng, jitter):
    """n sites of an x-fastest lattice, nx by ny a layer (the last layer ragged), jittered."""
    k = np.arange(n)
    base = np.stack([k % nx, (k // nx) % ny, k // (nx * ny)], axis=1) + 0.5
    return base * pitch + rng.uniform(-jitter, jitter, (n, 3))


def _bed_scene(case, seed):
    """A packed bed in a closed box: lattice neighbours overlap by about 1 %, so every grain starts
    in contact with its six neighbours, as in a settled pile (some three contacts a grain)."""
    from peclet.dem import workloads as W
    rng = np.random.default_rng(seed)
    if case.get("settled"):
        sc = W.plain_settled()
        sc.vel = sc.vel + rng.uniform(-1e-3, 1e-3, sc.vel.shape)
        return sc
    n = case["n"]
    nx = max(2, math.ceil(n ** (1.0 / 3.0) - 1e-9))
    a = 1.98 * R0
    pos = _lattice(n, nx, nx, a, rng, 0.02 * R0)
    m, inertia = _inertia(R0)
    mx = (nx * a, nx * a, (n // (nx * nx) + 3) * a)
    return W.Scene(name="bed", pos=pos, vel=rng.uniform(-0.05, 0.05, (n, 3)), inv_mass=np.full(n, 1.0 / m),
                   inv_inertia=np.full((n, 3), 1.0 / inertia), global_scale=R0,
                   domain=((0.0, 0.0, 0.0), mx, (False, False, False)), planes=W.box_planes((0.0, 0.0, 0.0), mx),
                   material=(0.5, 0.0, 0.5), iterations=(10, 10), dt=1e-5, substeps=10)


def _poly_radii(rng, n, top):
    return np.clip(rng.lognormal(np.log(R0), 0.25, n), 0.5 * R0, top)


def _periodic_scene(case, seed):
    """Lognormal radii on a jittered lattice, periodic in x and y, on a floor; the large neighbours
    touch."""
    from peclet.dem import workloads as W
    rng = np.random.default_rng(seed)
    n = case["n"]
    nx = max(4, math.ceil(n ** (1.0 / 3.0) - 1e-9))
    a = 2.15 * R0
    pos = _lattice(n, nx, nx, a, rng, 0.03 * R0)
    r = _poly_radii(rng, n, 1.08 * R0)
    m, inertia = _inertia(r)
    mx = (nx * a, nx * a, (n // (nx * nx) + 3) * a)
    return W.Scene(name="periodic", pos=pos, vel=rng.uniform(-0.05, 0.05, (n, 3)), inv_mass=1.0 / m,
                   inv_inertia=np.repeat(1.0 / inertia[:, None], 3, 1), scales=r / R0, global_scale=R0,
                   domain=((0.0, 0.0, 0.0), mx, (True, True, False)), planes=[(0.0, 0.0, 0.0, 0.0, 0.0, 1.0)],
                   material=(0.6, 0.0, 0.4), iterations=(10, 10), dt=2e-6, substeps=10)


def _drum_scenes(case, seed):
    """Uneven drums (R 50 mm, L 20 mm), each with a bed of touching grains at its bottom."""
    from peclet.dem import workloads as W
    rng = np.random.default_rng(seed)
    sizes = np.random.default_rng(case["scenes"])  # the scenes' sizes belong to the case, not to the seed
    R, L, a = 50e-3, 20e-3, 2.0 * R0
    grid = W.drum_wall_grid(R, L, 1e-3)
    g = np.stack(np.meshgrid(np.arange(10), np.arange(50), np.arange(50), indexing="ij"), -1).reshape(-1, 3)
    site = (g[:, [2, 1, 0]] + 0.5) * a + np.array([-R, -R, 0.0])
    site = site[np.hypot(site[:, 0], site[:, 1]) < R - 1.1 * R0]
    out, extras = [], []
    for s in range(case["scenes"]):
        omega, mu, e = rng.uniform(0.5, 3.0), rng.uniform(0.2, 0.8), rng.uniform(0.3, 0.9)
        n = min(int(sizes.integers(case["nmin"], case["nmax"] + 1)), len(site) // 2)
        order = np.argsort(site[:, 1], kind="stable")[:n]  # the lowest sites: a bed
        pos = site[np.sort(order)] + rng.uniform(-0.02 * R0, 0.02 * R0, (n, 3))
        r = rng.uniform(0.9 * R0, 1.01 * R0, n)
        m, inertia = _inertia(r)
        vel = rng.uniform(-0.05, 0.05, (n, 3))
        out.append(W.Scene(name=f"drum{s}", pos=pos, vel=vel, inv_mass=1.0 / m,
                           inv_inertia=np.repeat(1.0 / inertia[:, None], 3, 1), scales=r / R0, global_scale=R0,
                           domain=((-R, -R, 0.0), (R, R, L), (False, False, False)), gravity=(0.0, -9.81, 0.0),
                           material=(e, 0.0, mu), iterations=(10, 10), dt=5e-6, substeps=10))

        def extra(sim, w=omega):
            wid = sim.add_sdf_wall(*grid, 0.5, 0.5)
            sim.set_wall_velocity(wid, (0.0, 0.0, 0.0), (0.0, 0.0, w), (0.0, 0.0, 0.0))
        extras.append(extra)
    return out, extras


def _shell_scene(case, seed):
    """Hollow cylinders (outer radius 1 mm, length 3 mm, body axis y) stacked side by side with a small
    random tilt and a random spin about their axes, in a closed box, with a stratified point shell:
    each touches its neighbours along lines of shell points."""
    from peclet.dem import workloads as W
    rng = np.random.default_rng(seed)
    n = case["n"]
    r_out, r_in, length = 1e-3, 0.6e-3, 3e-3
    nx = max(2, math.ceil(n ** (1.0 / 3.0) - 1e-9))
    pitch = np.array([2.0e-3, 3.1e-3, 2.0e-3])
    k = np.arange(n)
    pos = (np.stack([k % nx, (k // nx) % nx, k // (nx * nx)], 1) + 0.5) * pitch + rng.uniform(-1e-5, 1e-5, (n, 3))
    half, spin = rng.normal(0.0, 0.005, (n, 2)), rng.uniform(0.0, np.pi, n)
    quat = np.stack([half[:, 0], np.sin(spin), half[:, 1], np.cos(spin)], 1)  # spin about y, tilted
    quat /= np.linalg.norm(quat, axis=1, keepdims=True)
    m = 1200.0 * np.pi * (r_out ** 2 - r_in ** 2) * length
    term = r_out ** 2 + r_in ** 2
    ixx, iyy = m * (3 * term + length ** 2) / 12.0, 0.5 * m * term
    mx = tuple(np.array([nx, nx, n // (nx * nx) + 2]) * pitch)
    return W.Scene(name="shells", pos=pos, vel=rng.uniform(-0.05, 0.05, (n, 3)), inv_mass=np.full(n, 1.0 / m),
                   inv_inertia=np.tile([1.0 / ixx, 1.0 / iyy, 1.0 / ixx], (n, 1)), quat=quat,
                   shape=(W.HOLLOW_CYLINDER, 1.0, length / r_out, (r_out - r_in) / r_out), global_scale=r_out,
                   domain=((0.0, 0.0, 0.0), mx, (False, False, False)), planes=W.box_planes((0.0, 0.0, 0.0), mx),
                   material=(0.4, 0.0, 0.3), iterations=(20, 10), dt=5e-5 / 8, substeps=8,
                   shell=W.hollow_cylinder_shell(case["points"], seed=seed))


def _hertz_inputs(case, seed):
    """Lognormal spheres on a jittered lattice in an SDF-wall box; velocities +-0.5 m/s."""
    from peclet.dem import workloads as W
    rng = np.random.default_rng(seed)
    n = case["n"]
    nx = max(3, math.ceil(n ** (1.0 / 3.0) - 1e-9))
    a = 2.15 * R0
    pos = _lattice(n, nx, nx, a, rng, 0.03 * R0)
    r = _poly_radii(rng, n, 1.08 * R0)
    L, H = nx * a, (n // (nx * nx) + 3) * a
    return {"pos": pos, "vel": rng.uniform(-0.5, 0.5, (n, 3)), "r": r, "L": L, "H": H, "dt": 2e-6,
            "grid": W.box_wall_grid(L, H)}


def _calibration_inputs(case, seed):
    """Boxes of r = 1 mm spheres on a jittered lattice with gaps, +-0.2 m/s, six shared planes, and
    seeded target positions."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    per = nx * ny * nz
    pitch = np.array([2.5, 2.5, 2.5]) * R0
    box = pitch * np.array([nx, ny, nz])
    c = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 3)
    n = case["scenes"] * per
    x0 = np.tile((c + 0.5) * pitch, (case["scenes"], 1)) + rng.uniform(-0.1e-3, 0.1e-3, (n, 3))
    planes = [[0, 0, 0, 1, 0, 0], [box[0], 0, 0, -1, 0, 0], [0, 0, 0, 0, 1, 0], [0, box[1], 0, 0, -1, 0],
              [0, 0, 0, 0, 0, 1], [0, 0, box[2], 0, 0, -1]]
    return {"x0": x0, "v0": rng.uniform(-0.2, 0.2, (n, 3)), "w0": np.zeros((n, 3)), "planes": planes,
            "first": np.arange(case["scenes"] + 1) * per, "target": x0 + rng.normal(size=(n, 3)) * 1e-3, "dt": 2e-5}


# ---- the calls ------------------------------------------------------------------------------------
def _pinned(n, cols):
    return torch.zeros((n, cols), dtype=torch.float64, pin_memory=True).numpy()


def prepare(case, seed):
    import peclet.dem as dem
    kind = case["kind"]
    if kind in ("bed", "periodic", "shells"):
        sc = {"bed": _bed_scene, "periodic": _periodic_scene, "shells": _shell_scene}[kind](case, seed)
        sim = sc.apply(dem.Simulation(sc.n + 8, case["precision"]))
        start = None
        if kind != "periodic":
            quat = sc.quat if sc.quat is not None else np.tile([0.0, 0.0, 0.0, 1.0], (sc.n, 1))
            start = {"set_positions": sc.pos, "set_quaternions": quat, "set_velocities": sc.vel,
                     "set_angular_velocities": sc.angvel if sc.angvel is not None else np.zeros((sc.n, 3)),
                     "set_inv_mass": sc.inv_mass, "set_inv_inertia": sc.inv_inertia}
        return {"kind": "step", "sim": sim, "dt": sc.dt, "substeps": sc.substeps, "start": start,
                "out": [_pinned(sc.n, k) for k in (3, 3, 4, 3)]}
    if kind == "drums":
        from peclet.dem.batch import apply_batch
        scenes, extras = _drum_scenes(case, seed)
        n = sum(s.n for s in scenes)
        sim = dem.Simulation(n + 8, case["precision"])
        apply_batch(sim, scenes, extras)
        return {"kind": "step", "sim": sim, "dt": scenes[0].dt, "substeps": scenes[0].substeps, "start": None,
                "out": [_pinned(n, k) for k in (3, 3, 4, 3)]}
    if kind == "hertz":
        h = _hertz_inputs(case, seed)
        n = case["n"]
        m, inertia = _inertia(h["r"])
        sim = dem.Simulation(n + 8, case["precision"])
        sim.initialize_shape(1, 1.0)
        sim.set_global_scale(R0)
        sim.set_domain((0.0, 0.0, 0.0), (h["L"], h["L"], h["H"]))
        sim.enable_periodicity(False, False, False)
        sim.set_gravity(0.0, 0.0, -9.81)
        sim.set_material_params(HZ["e"], 0.0, HZ["mu"])
        sim.set_hertz_material(0, HZ["youngs"], HZ["poisson"])
        sim.set_positions(h["pos"])
        sim.set_scales(h["r"] / R0)
        sim.set_velocities(h["vel"])
        sim.set_inv_mass(1.0 / m)
        sim.set_inv_inertia(np.repeat(1.0 / inertia[:, None], 3, 1))
        sim.add_sdf_wall(*h["grid"], HZ["e"], HZ["mu"])
        return {"kind": "hertz", "sim": sim, "dt": h["dt"], "substeps": case["substeps"],
                "out": [_pinned(n, 3) for _ in range(3)]}
    if kind == "calibration":
        from peclet.dem.adjoint import HertzSpheres
        c = _calibration_inputs(case, seed)
        n = len(c["x0"])
        m, inertia = _inertia(np.full(n, R0))
        sim = HertzSpheres(np.full(n, R0), m, inertia, c["first"], c["planes"], 0.3, c["dt"], (0.0, 0.0, -9.81),
                           case["precision"], 100)
        t = lambda a: torch.as_tensor(a, dtype=sim.dtype, device="cuda")
        return {"kind": "calibration", "sim": sim, "x0": t(c["x0"]), "v0": t(c["v0"]), "w0": t(c["w0"]),
                "target": torch.as_tensor(c["target"], device="cuda"), "substeps": case["substeps"]}
    from peclet.dem.xpbd_adjoint import XpbdRollout
    sc = _bed_scene(case, seed)
    sc.material = (0.5, 0.3, 0.5)
    sim = sc.apply(dem.Simulation(sc.n + 8, "fp64"))
    rng = np.random.default_rng(seed + 1)
    t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device="cuda")
    start = [t(sc.pos), t(np.tile([0.0, 0.0, 0.0, 1.0], (sc.n, 1))), t(sc.vel), t(np.zeros((sc.n, 3)))]
    return {"kind": "xpbd_adjoint", "roll": XpbdRollout(sim), "start": start, "material": sc.material,
            "weights": [t(rng.normal(size=tuple(s.shape))) for s in start], "substeps": case["substeps"]}


def run(state):
    kind = state["kind"]
    if kind in ("step", "hertz"):
        sim, dt = state["sim"], state["dt"]
        if kind == "hertz":
            sim.step_hertz(dt, state["substeps"])
            px, pv, pw = state["out"]
            return sim.get_positions(out=px), sim.get_velocities(out=pv), sim.get_angular_velocities(out=pw)
        for setter, rows in (state["start"] or {}).items():
            getattr(sim, setter)(rows)
        for _ in range(state["substeps"]):
            sim.step(dt)
        px, pv, pq, pw = state["out"]
        return (sim.get_positions(out=px), sim.get_velocities(out=pv), sim.get_quaternions(out=pq),
                sim.get_angular_velocities(out=pw))
    if kind == "calibration":
        sim = state["sim"]
        theta = torch.tensor(THETA, dtype=torch.float64, requires_grad=True)
        v0 = state["v0"].clone().requires_grad_(True)
        x, v, w = sim.rollout(state["x0"], v0, state["w0"], theta, state["substeps"])
        ((x.double() - state["target"]) ** 2).sum().backward()
        return {"x": x.detach(), "v": v.detach(), "w": w.detach(), "dtheta_E": theta.grad[:1],
                "dtheta_emu": theta.grad[1:], "dv0": v0.grad}
    start = [s.clone().requires_grad_(True) for s in state["start"]]
    theta = torch.tensor(state["material"], dtype=torch.float64, requires_grad=True)
    out = state["roll"](*start, theta, state["substeps"])
    sum((a * b).sum() for a, b in zip(out, state["weights"])).backward()
    return {"end": [o.detach() for o in out], "dstart": [s.grad for s in start], "dtheta": theta.grad}


# ---- cost and tolerance -----------------------------------------------------------------------------
def _bodies(case):
    if case["kind"] == "drums":
        return int(case["scenes"] * 0.5 * (case["nmin"] + min(case["nmax"], 8900)))
    if case["kind"] == "calibration":
        return case["scenes"] * case["nx"] * case["ny"] * case["nz"]
    return case["n"]


def work(case):
    """Bytes: the state (13 values a body) and the body constants (5) read, the state written, once a
    substep, and each contact's 20 values once. Flops: one velocity update of some 450 operations a
    contact and sweep, a position update of some 150, a Hertz contact of some 200, an integration of
    some 60 a body; an adjoint twice its forward."""
    n, kind = _bodies(case), case["kind"]
    size = 4 if case.get("precision") in ("fp32", "mixed") else 8
    subs = case.get("substeps", 8 if kind == "shells" else 10)
    contacts = {"bed": 3.0, "drums": 2.0, "xpbd_adjoint": 3.0, "periodic": 0.4, "shells": 40.0, "hertz": 0.4,
                "calibration": 0.02}[kind] * n
    sweeps = {"bed": 30, "drums": 20, "xpbd_adjoint": 30, "periodic": 5, "shells": 10}.get(kind, 0)
    per = 31 * n + 20 * contacts
    flops = 60 * n + contacts * (450 * sweeps + 150 * 5 if sweeps else 200)
    if kind == "shells":  # two pairs a body, each way every shell point against the other's surface
        flops += 4.0 * n * 60.0 * case["points"]
    factor = 3 if kind in ("calibration", "xpbd_adjoint") else 1
    return {"bytes": float(per * size * subs * factor), "flops": float(flops * subs * factor)}


def tolerance(case):
    """The float and mixed XPBD steps and the float Hertz engine define their result bit for bit (the
    serial order of the reference's float arithmetic, canonical on every launch shape). In double the
    same order in another rounding moves a result by some 1e-14 a substep."""
    kind = case["kind"]
    if kind == "calibration":
        return {"rel": 1e-4} if case["precision"] == "fp32" else {"rel": 1e-8}
    if kind == "xpbd_adjoint":
        return {"rel": 1e-8}
    if case["precision"] != "fp64":
        return "exact"
    return {"rel": 1e-10}


# ---- the Hertz substep in plain torch, 64 bits --------------------------------------------------------
def _pairs(x, r, scene, skin):
    """All pairs i < j of one scene with a gap below skin, by a cell list."""
    side = float(2 * r.max()) + skin
    lo = x.min(dim=0).values
    c = ((x - lo) / side).long() + 1
    dims = c.max(dim=0).values + 2
    cell = ((scene * dims[2] + c[:, 2]) * dims[1] + c[:, 1]) * dims[0] + c[:, 0]
    key, order = torch.sort(cell)
    out = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            base = cell + (dz * dims[1] + dy) * dims[0]
            a, b = torch.searchsorted(key, base - 1), torch.searchsorted(key, base + 1, right=True)
            i = torch.repeat_interleave(torch.arange(len(x), device=x.device), b - a)
            first = torch.repeat_interleave(a - (torch.cumsum(b - a, 0) - (b - a)), b - a)
            j = order[first + torch.arange(len(i), device=x.device)]
            keep = (i < j) & (scene[i] == scene[j])
            i, j = i[keep], j[keep]
            near = (x[i] - x[j]).norm(dim=1) < r[i] + r[j] + skin
            out.append(torch.stack([i[near], j[near]], 1))
    p = torch.cat(out)
    return p[torch.argsort(p[:, 0] * len(x) + p[:, 1])]


def _hertz_contact(delta, nh, vr, r_star, m_star, e_mod, nu, e, mu, dt, xi):
    """Hertz-Mindlin force of touching contacts (delta > 0) and their new tangential history."""
    e_star = e_mod / (2 * (1 - nu * nu))
    g_star = e_mod / (4 * (2 - nu) * (1 + nu))
    root = torch.sqrt(r_star * delta)
    sn, st = 2 * e_star * root, 8 * g_star * root
    le = torch.log(e)
    beta = le / torch.sqrt(le * le + 9.8696044)
    eta_n, eta_t = -2 * 0.9128709 * beta * torch.sqrt(sn * m_star), -2 * 0.9128709 * beta * torch.sqrt(st * m_star)
    vn = (vr * nh).sum(1)
    fs = 4.0 / 3.0 * e_star * root * delta
    vt = vr - nh * vn[:, None]
    xi = xi + vt * dt
    xi = xi - nh * (xi * nh).sum(1, keepdim=True)
    ft = -st[:, None] * xi - eta_t[:, None] * vt
    sq = (ft * ft).sum(1)
    fl = torch.sqrt(torch.where(sq > 0, sq, torch.ones_like(sq))) * (sq > 0)
    fm = mu * fs
    slip = fl > fm
    ft_s = ft * (fm / torch.where(slip, fl, torch.ones_like(fl)))[:, None]
    xi = torch.where(slip[:, None], -(ft_s + eta_t[:, None] * vt) / st[:, None], xi)
    return nh * (fs - eta_n * vn)[:, None] + torch.where(slip[:, None], ft_s, ft), xi


def _wall_distance(p, grid, shape, origin, h):
    """Trilinear sample of the container grid, clamped, minus the distance to the grid's box."""
    f = (p - origin) / h
    top = torch.tensor([s - 1 for s in shape], dtype=p.dtype, device=p.device)
    c = torch.minimum(torch.clamp(f, min=0.0), top)
    i0 = c.long()
    i1 = torch.minimum(i0 + 1, top.long())
    t = c - i0
    at = lambda a, b, d: grid[d[:, 2], b[:, 1], a[:, 0]]
    mix = lambda u, v, w: u * (1 - w) + v * w
    c0 = mix(mix(at(i0, i0, i0), at(i1, i0, i0), t[:, 0]), mix(at(i0, i1, i0), at(i1, i1, i0), t[:, 0]), t[:, 1])
    c1 = mix(mix(at(i0, i0, i1), at(i1, i0, i1), t[:, 0]), mix(at(i0, i1, i1), at(i1, i1, i1), t[:, 0]), t[:, 1])
    return mix(c0, c1, t[:, 2]) - ((f - c) * h).norm(dim=1)


def _touching(x, v, w, r, inv_m, inv_i, pairs, xi, law, e, mu, dt):
    """Pair forces and torques on every body, and the new pair histories (zero where apart)."""
    i, j = pairs[:, 0], pairs[:, 1]
    gap = (x[i] - x[j]).detach().norm(dim=1) - r[i] - r[j]
    on = gap < 0
    i, j = i[on], j[on]
    dx = x[i] - x[j]
    d = dx.norm(dim=1)
    delta = r[i] + r[j] - d
    nh = dx / d[:, None]
    ra, rb = -nh * (r[i] - 0.5 * delta)[:, None], nh * (r[j] - 0.5 * delta)[:, None]
    vr = v[i] + torch.cross(w[i], ra, dim=1) - v[j] - torch.cross(w[j], rb, dim=1)
    f, new = _hertz_contact(delta, nh, vr, r[i] * r[j] / (r[i] + r[j]), 1 / (inv_m[i] + inv_m[j]), *law, e, mu, dt,
                            xi[on])
    F = torch.zeros_like(x).index_add(0, i, f).index_add(0, j, -f)
    T = torch.zeros_like(x).index_add(0, i, torch.cross(ra, f, dim=1)).index_add(0, j, torch.cross(rb, -f, dim=1))
    return F, T, torch.zeros_like(xi).index_put((on.nonzero()[:, 0],), new)


def _single_sided(x, v, w, r, inv_m, dist, normal, xi, law, e, mu, dt):
    """Forces and torques of the spheres on one container at rest: distance and unit normal given."""
    on = (r - dist.detach()) > 0
    k = on.nonzero()[:, 0]
    delta, nh = (r - dist)[k], normal[k]
    ra = -nh * (r[k] - 0.5 * delta)[:, None]
    vr = v[k] + torch.cross(w[k], ra, dim=1)
    f, new = _hertz_contact(delta, nh, vr, r[k], 1 / inv_m[k], *law, e, mu, dt, xi[k])
    return (torch.zeros_like(x).index_add(0, k, f), torch.zeros_like(x).index_add(0, k, torch.cross(ra, f, dim=1)),
            torch.zeros_like(xi).index_put((k,), new))


def _relist(pairs, xi, new, n):
    """The histories of the new pair list: those of the old one by pair, zero for the others."""
    old_key, key = pairs[:, 0] * n + pairs[:, 1], new[:, 0] * n + new[:, 1]
    if not len(old_key) or not len(key):
        return torch.zeros((len(key), 3), dtype=torch.float64, device=new.device)
    at = torch.searchsorted(old_key, key).clamp(max=len(old_key) - 1)
    return torch.where((old_key[at] == key)[:, None], xi[at], torch.zeros_like(xi[at]))


def exact(case, seed):
    """The explicit Hertz paths in 64 bits. The XPBD step has no value of its own to compare with: its
    result is defined by the order of its Gauss-Seidel updates, so those cases give None."""
    if case["kind"] not in ("hertz", "calibration"):
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    t = lambda a: torch.as_tensor(np.asarray(a, np.float64), device=dev)
    g = t([0.0, 0.0, -9.81])
    if case["kind"] == "hertz":
        h = _hertz_inputs(case, seed)
        n, r = case["n"], t(h["r"])
        m, inertia = _inertia(r)
        x, v, w = t(h["pos"]), t(h["vel"]), torch.zeros((n, 3), dtype=torch.float64, device=dev)
        grid, nx, ny, nz, origin, spacing = h["grid"]
        grid, origin, hs = t(grid).reshape(nz, ny, nx), t(origin), t(spacing)
        e, mu, law = t(HZ["e"]), t(HZ["mu"]), (t(HZ["youngs"]), HZ["poisson"])
        scene = torch.zeros(n, dtype=torch.long, device=dev)
        pairs, xi = torch.zeros((0, 2), dtype=torch.long, device=dev), torch.zeros((0, 3), dtype=torch.float64, device=dev)
        xi_w = torch.zeros((n, 3), dtype=torch.float64, device=dev)
        half = 0.5 * float(spacing[0])
        for k in range(case["substeps"]):
            if k % 50 == 0:  # 50 substeps of 2e-6 s at a few m/s stay well inside the skin
                new = _pairs(x, r, scene, 1.0 * R0)
                pairs, xi = new, _relist(pairs, xi, new, n)
            F, T, xi = _touching(x, v, w, r, 1 / m, 1 / inertia, pairs, xi, law, e, mu, h["dt"])
            sample = lambda p: _wall_distance(p, grid, (nx, ny, nz), origin, hs)
            eye = torch.eye(3, dtype=torch.float64, device=dev) * half
            grad = torch.stack([sample(x + eye[a]) - sample(x - eye[a]) for a in range(3)], 1)
            normal = grad / grad.norm(dim=1, keepdim=True).clamp(min=1e-12)
            Fw, Tw, xi_w = _single_sided(x, v, w, r, 1 / m, sample(x), normal, xi_w, law, e, mu, h["dt"])
            v = v + ((F + Fw) / m[:, None] + g) * h["dt"]
            w = w + (T + Tw) / inertia[:, None] * h["dt"]
            x = x + v * h["dt"]
        return x, v, w
    n = _bodies(case)
    if n * case["substeps"] > 8e6:  # the recorded graph would not fit
        return None
    c = _calibration_inputs(case, seed)
    f32 = case["precision"] == "fp32"
    rnd = (lambda a: t(np.asarray(a, np.float32))) if f32 else t  # the inputs as the call takes them
    r = torch.full((n,), R0, dtype=torch.float64, device=dev)
    m, inertia = _inertia(r)
    theta = torch.tensor(THETA, dtype=torch.float64, device=dev, requires_grad=True)
    v0 = rnd(c["v0"]).requires_grad_(True)
    x, v, w = rnd(c["x0"]), v0, rnd(c["w0"])
    scene = torch.repeat_interleave(torch.arange(case["scenes"], device=dev), n // case["scenes"])
    planes = t(c["planes"])
    pairs, xi = torch.zeros((0, 2), dtype=torch.long, device=dev), torch.zeros((0, 3), dtype=torch.float64, device=dev)
    xi_w = [torch.zeros((n, 3), dtype=torch.float64, device=dev) for _ in planes]
    for k in range(case["substeps"]):
        if k % 20 == 0:
            new = _pairs(x.detach(), r, scene, 0.6 * R0)
            pairs, xi = new, _relist(pairs, xi, new, n)
        law = (theta[0], 0.3)
        F, T, xi = _touching(x, v, w, r, 1 / m, 1 / inertia, pairs, xi, law, theta[1], theta[2], c["dt"])
        for p in range(len(planes)):
            dist = ((x - planes[p, :3]) * planes[p, 3:]).sum(1)
            Fw, Tw, xi_w[p] = _single_sided(x, v, w, r, 1 / m, dist, planes[p, 3:].expand(n, 3), xi_w[p], law, theta[1],
                                            theta[2], c["dt"])
            F, T = F + Fw, T + Tw
        v = v + (F / m[:, None] + g) * c["dt"]
        w = w + T / inertia[:, None] * c["dt"]
        x = x + v * c["dt"]
    ((x - t(c["target"])) ** 2).sum().backward()
    # a float rollout meets contact onsets at other instants: its gradients are those of another
    # smooth piece for the grains at an onset, and have no 64-bit value to compare with
    return {"x": x.detach(), "v": v.detach(), "w": w.detach(), "dtheta_E": None if f32 else theta.grad[:1],
            "dtheta_emu": None if f32 else theta.grad[1:], "dv0": None if f32 else v0.grad}
