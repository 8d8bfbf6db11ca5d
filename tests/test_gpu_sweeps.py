"""The sweep loops' launch forms against the oracle, at the sizes where they change: the flow of body
states in one cluster (1 to 16 blocks) and on the grid, ragged last warps, single bodies, a body in
contact with its own periodic image, an adaptive stop after the first sweep and one sweep only; and the
dense position sweeps (saturated and uncoloured contacts) in one block and on the grid. Bit-exact at
float; 1e-12 relative at double, the step's own bar."""
import numpy as np
import pytest

import parity as P
import scenes as S
from peclet.dem import workloads as W

pytestmark = pytest.mark.gpu

PRECISIONS = [("fp32", 0.0), ("fp64", 1e-12)]


def _compare(gpu_api, orc_api, sc, steps, precision, rtol):
    a, b = P.build(gpu_api, sc, None, precision), P.build(orc_api, sc, None, precision)
    for k in range(steps):
        a.step(sc.dt)
        b.step(sc.dt)
        bad = P.diff(P.snapshot(a), P.snapshot(b), rtol=rtol)
        assert not bad, f"substep {k}: {bad[:4]}"
    return a


def _bed(n, iters=(10, 10), seed=41):
    """The first n spheres of a touching lattice column on the floor."""
    nx = max(1, round(n ** (1 / 3)))
    sc = W.plain_settling(seed=seed, nx=nx, ny=nx, nz=-(-n // (nx * nx)), cells_z=n // (nx * nx) + 3, spacing_r=1.98,
                          jitter_r=0.02, vmax=0.05, iterations=iters)
    sc.pos, sc.vel, sc.inv_mass, sc.inv_inertia = (a[:n].copy() for a in (sc.pos, sc.vel, sc.inv_mass, sc.inv_inertia))
    return sc


@pytest.mark.parametrize("precision,rtol", PRECISIONS)
@pytest.mark.parametrize("entries", [None, 0], ids=["cluster", "grid"])
@pytest.mark.parametrize("n,iters", [(1, (10, 10)), (2, (10, 10)), (65, (1, 1)), (700, (3, 10)), (2500, (10, 4))])
def test_flow_forms(gpu_api, orc_api, monkeypatch, n, iters, entries, precision, rtol):
    if entries is not None:
        monkeypatch.setenv("PDEM_SWEEP_CLUSTER_ENTRIES", str(entries))
    _compare(gpu_api, orc_api, _bed(n, iters), 3, precision, rtol)


@pytest.mark.parametrize("precision,rtol", PRECISIONS)
@pytest.mark.parametrize("seed", [3, 4, 5])
def test_flow_own_image(gpu_api, orc_api, monkeypatch, seed, precision, rtol):
    """Spheres stacked in a box periodic in x that is narrower than a sphere: each touches its own image
    (one body on both sides of a manifold). The first substep, whose sweeps start from the bodies' velocities,
    against the oracle; the next ones, warm-started, by the cluster and by the grid, which give the same bits."""
    r, L = 1e-3, 1.995e-3
    rng = np.random.default_rng(seed)
    pos = np.stack([np.full(5, 0.5 * L), np.full(5, r), r * (0.99 + 1.98 * np.arange(5))], 1)
    im, inertia = W.sphere_props(r, 2500.0)
    sc = W.Scene(name="own_image", pos=pos, vel=rng.uniform(-0.05, 0.05, (5, 3)), inv_mass=np.full(5, im),
                 inv_inertia=np.full((5, 3), inertia), global_scale=r,
                 domain=((0, 0, 0), (L, 3 * r, 14 * r), (True, False, False)), planes=[(0, 0, 0, 0, 0, 1)],
                 material=(0.5, 0.0, 0.5), dt=1e-5)
    a = _compare(gpu_api, orc_api, sc, 1, precision, rtol)
    assert a.counters()["manifolds"] > 5
    monkeypatch.setenv("PDEM_SWEEP_CLUSTER_ENTRIES", "0")
    b = _compare(gpu_api, orc_api, sc, 1, precision, rtol)
    for _ in range(3):
        a.step(sc.dt)
        b.step(sc.dt)
        assert not P.diff(P.snapshot(a), P.snapshot(b))


def test_flow_tags_start_again(gpu_api, orc_api, monkeypatch):
    """The mailbox tags of the grid form are numbered through a simulation's launches, as many a launch as it
    may sweep, and start again when 32 bits are used up: with 0x0f000000 sweeps allowed (of which two spheres
    on a floor take a few, so that 50 give the same bits) that is within 24 substeps."""
    monkeypatch.setenv("PDEM_SWEEP_CLUSTER_ENTRIES", "0")
    a, b = P.build(gpu_api, _bed(2, (10, 0x0F000000)), None, "fp32"), P.build(orc_api, _bed(2, (10, 50)), None, "fp32")
    for k in range(24):
        a.step(1e-5)
        b.step(1e-5)
        bad = P.diff(P.snapshot(a), P.snapshot(b))
        assert not bad, f"substep {k}: {bad[:4]}"


def _grain(touching, radius=1e-3):
    """One large grain, the last body, covered by `touching` small ones that press on it."""
    k = np.arange(touching) + 0.5
    phi, theta = np.arccos(1 - 2 * k / touching), np.pi * (1 + 5 ** 0.5) * k
    u = np.stack([np.cos(theta) * np.sin(phi), np.sin(theta) * np.sin(phi), np.cos(phi)], 1)
    rho = (touching * 4.6 / (4 * np.pi)) ** 0.5 - 1
    L = 2 * (rho + 3) * radius
    pos = np.concatenate([L / 2 + u * (rho + 0.99) * radius, [[L / 2] * 3]])
    r = np.full(touching + 1, radius)
    r[-1] = rho * radius
    im, inertia = W.sphere_props(r, 2500.0)
    rng = np.random.default_rng(touching)
    return W.Scene(name="grain", pos=pos, vel=np.concatenate([-0.5 * u, [[0.0] * 3]]) + rng.uniform(-0.1, 0.1, pos.shape),
                   inv_mass=im, inv_inertia=np.repeat(np.asarray(inertia)[:, None], 3, 1), scales=r / radius,
                   global_scale=radius, domain=((0, 0, 0), (L, L, L), (False,) * 3),
                   planes=W.box_planes((0, 0, 0), (L, L, L)), material=(0.5, 0.0, 0.5), dt=1e-5)


@pytest.mark.parametrize("precision,rtol", PRECISIONS)
@pytest.mark.parametrize("entries", [None, 0], ids=["cluster", "grid"])
@pytest.mark.parametrize("touching,colours", [(62, 62), (63, 63), (200, 63)])
def test_saturated_manifolds(gpu_api, orc_api, monkeypatch, touching, colours, entries, precision, rtol):
    """A grain of more touching neighbours than colours: the velocity loops take the saturated colour in
    manifold order, from the packed records in one cluster or on the grid."""
    if entries is not None:
        monkeypatch.setenv("PDEM_SWEEP_CLUSTER_ENTRIES", str(entries))
    sc = _grain(touching)
    a, b = P.build(gpu_api, sc, None, precision), P.build(orc_api, sc, None, precision)
    for k in range(2):
        a.step(sc.dt)
        b.step(sc.dt)
        bad = P.diff(P.snapshot(a), P.snapshot(b), rtol=rtol)
        assert not bad, f"substep {k}: {bad[:4]}"
        if k == 0:
            assert a.counters()["colors_velocity"] == colours


@pytest.mark.parametrize("precision,rtol", PRECISIONS)
@pytest.mark.parametrize("entries", [None, 0], ids=["cluster", "grid"])
def test_flow_of_many_colours(gpu_api, orc_api, monkeypatch, entries, precision, rtol):
    """100 grains of 43 touching neighbours: some 100 entries a colour, whose mailboxes in double need more
    blocks than the entries of a colour ask for."""
    if entries is not None:
        monkeypatch.setenv("PDEM_SWEEP_CLUSTER_ENTRIES", str(entries))
    one, n = _grain(43), 100
    L = np.array(one.domain[1])
    sc = _grain(43)
    sc.pos = np.concatenate([one.pos + L * [k % 10, k // 10, 0] for k in range(n)])
    for k in ("vel", "inv_mass", "inv_inertia", "scales"):
        setattr(sc, k, np.concatenate([getattr(one, k)] * n))
    sc.domain = ((0, 0, 0), tuple(L * [10, 10, 1]), (False,) * 3)
    sc.planes = W.box_planes(*sc.domain[:2])
    a, b = P.build(gpu_api, sc, None, precision), P.build(orc_api, sc, None, precision)
    a.step(sc.dt)
    b.step(sc.dt)
    bad = P.diff(P.snapshot(a), P.snapshot(b), rtol=rtol)
    assert not bad, bad[:4]
    c = a.counters()
    assert c["colors_velocity"] >= 43 and c["manifolds"] >= 4300


@pytest.mark.parametrize("entries", [None, 0], ids=["cluster", "grid"])
def test_flow_time_out(gpu_api, orc_api, monkeypatch, entries):
    """Every wait of the flow for another block gives up after one poll (a state, the sweep's maximum): no
    wait is repeated after that, so a loop of 600 sweeps ends at once, the step reports the error, and with
    the default limit the next substeps match the oracle."""
    import time
    if entries is not None:
        monkeypatch.setenv("PDEM_SWEEP_CLUSTER_ENTRIES", str(entries))
    sc = _bed(700, (10, 600))
    sim = P.build(gpu_api, sc, None, "fp64")
    sim.debug_set_barrier_spins(1)
    t = time.monotonic()
    with pytest.raises(RuntimeError, match="barrier"):
        for _ in range(3):
            sim.step(sc.dt)
    assert time.monotonic() - t < 5.0  # 600 sweeps of some 10 items at a microsecond or two, and the launches
    sim.debug_set_barrier_spins(0)
    sc.iterations = (10, 10)
    sim.set_solver_iterations(*sc.iterations)
    sim.set_positions(sc.pos)
    sim.set_velocities(sc.vel)
    sim.set_inv_mass(sc.inv_mass)
    sim.set_inv_inertia(sc.inv_inertia)
    ref = P.build(orc_api, sc, None, "fp64")
    for k in range(3):
        sim.step(sc.dt)
        ref.step(sc.dt)
        bad = P.diff(P.snapshot(sim), P.snapshot(ref), rtol=1e-12)
        assert not bad, f"after the time-out, substep {k}: {bad[:4]}"


def _stacked(n, points, seed=7):
    """Hollow cylinders side by side with a small tilt: tens of shell-point contacts a pair."""
    rng = np.random.default_rng(seed)
    nx = max(2, round(n ** (1 / 3)))
    pitch = np.array([2.0e-3, 3.1e-3, 2.0e-3])
    k = np.arange(n)
    sc = S.cylinders(seed=seed, n=n, shell=W.hollow_cylinder_shell(points, seed=seed))
    sc.pos = (np.stack([k % nx, k // (nx * nx), (k // nx) % nx], 1) + 0.5) * pitch + rng.uniform(-1e-5, 1e-5, (n, 3))
    half, spin = rng.normal(0.0, 0.005, (n, 2)), rng.uniform(0.0, np.pi, n)
    sc.quat = np.stack([half[:, 0], np.sin(spin), half[:, 1], np.cos(spin)], 1)
    sc.quat /= np.linalg.norm(sc.quat, axis=1, keepdims=True)
    mx = tuple(np.array([nx, n // (nx * nx) + 1, nx]) * pitch)
    sc.domain, sc.planes = ((0, 0, 0), mx, (False,) * 3), W.box_planes((0, 0, 0), mx)
    return sc


@pytest.mark.parametrize("precision,rtol", PRECISIONS)
@pytest.mark.parametrize("entries", [None, 0], ids=["block", "grid"])
@pytest.mark.parametrize("n,points,colours", [(2, 512, 0), (9, 256, 0), (120, 512, 63)])
def test_dense_forms(gpu_api, orc_api, monkeypatch, n, points, colours, entries, precision, rtol):
    if entries is not None:
        monkeypatch.setenv("PDEM_DENSE_ONE_ENTRIES", str(entries))
    sim = _compare(gpu_api, orc_api, _stacked(n, points), 2, precision, rtol)
    assert sim.counters()["colors_position"] >= colours


@pytest.mark.parametrize("precision,rtol", PRECISIONS)
@pytest.mark.parametrize("form", ["block", "cluster", "grid"])
@pytest.mark.parametrize("scene", ["grain63", "grain64", "grain300", "grains", "stacked120"])
def test_dense_forms_of_levels(gpu_api, orc_api, monkeypatch, scene, form, precision, rtol):
    """The saturated contacts in levels of one run (those of one large grain: one warp's outside the one-block
    form), of a few runs (one block's) and of many: two grains have levels of two runs and then of one, 120
    cylinders one of 45 and then fewer."""
    if form != "block":
        monkeypatch.setenv("PDEM_DENSE_ONE_ENTRIES", "0")
    if form == "grid":
        monkeypatch.setenv("PDEM_SWEEP_CLUSTER_ENTRIES", "0")
    if scene == "grains":
        sc, b = _grain(75), _grain(110)
        sc.domain = ((0, 0, 0), tuple(sc.domain[1][k] + b.domain[1][k] for k in range(3)), (False,) * 3)
        b.pos = b.pos + [float(sc.pos[-1, 0]) * 2, 0, 0]
        for k in ("pos", "vel", "inv_mass", "inv_inertia", "scales"):
            setattr(sc, k, np.concatenate([getattr(sc, k), getattr(b, k)]))
        sc.planes = W.box_planes(*sc.domain[:2])
    else:
        sc = _grain(int(scene[5:])) if scene.startswith("grain") else _stacked(120, 512)
    sim = _compare(gpu_api, orc_api, sc, 2, precision, rtol)
    assert sim.counters()["colors_position"] == 63


@pytest.mark.parametrize("form", ["shared", "cluster", "grid"])
@pytest.mark.parametrize("touching", [16, 17, 32, 33, 65, 300])
def test_colouring_forms(gpu_api, orc_api, monkeypatch, touching, form):
    """The colouring's rounds in shared memory, its visits without rounds in a cluster and on the grid, with
    lists sorted by eight lanes (up to 16 entries) or by items of 32: the oracle's colours, on a large grain (a
    chain as long as its list) and on a bed."""
    if form == "cluster":
        monkeypatch.setenv("PDEM_COLOR_ONE_BYTES", "0")
    if form == "grid":
        monkeypatch.setenv("PDEM_COLOR_CLUSTER_ENTRIES", "0")
    _compare(gpu_api, orc_api, _grain(touching), 2, "fp32", 0.0)
    _compare(gpu_api, orc_api, _bed(20 * touching), 1, "fp32", 0.0)


@pytest.mark.parametrize("precision,rtol", PRECISIONS)
@pytest.mark.parametrize("scene", ["bed", "reversed"])
def test_support_levels_on_the_grid(gpu_api, orc_api, monkeypatch, scene, precision, rtol):
    """The support levels computed by the whole grid (every graph sent there): a bed whose serial sweeps
    reach the fixed point, and a column numbered top to bottom whose sweeps stop short of it."""
    monkeypatch.setenv("PDEM_GROUND_ONE_BYTES", "0")
    _compare(gpu_api, orc_api, _bed(700) if scene == "bed" else S.reversed_column(), 12, precision, rtol)
