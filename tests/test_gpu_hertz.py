"""GPU parity of the explicit Hertz-Mindlin engine (`step_hertz`, src/sim.hpp:628-750) through the
C ABI: tangential history keys and vectors and the state after every call, against the oracle
restatement (bit-exact at float, within 1e-12 relative at double)."""
import numpy as np
import pytest

import parity as P
import scenes as S
from peclet.dem import workloads as W

pytestmark = pytest.mark.gpu


def _drum_spheres():
    sc, ex = S.spheres_in_drum()
    sc.planes = []

    def extra(s):
        ex(s)
        s.set_hertz_material(0, 1e7, 0.3)
    return sc, extra


def _dense_drum():
    sc, ex = S.spheres_in_drum(seed=21, n=240, omega=3.0)
    sc.planes = []

    def extra(s):
        ex(s)
        s.set_hertz_material(0, 5e6, 0.25)
    return sc, extra


def _shape_pairs():
    import hertz_cases as HC
    return HC.shape_pairs()


def _shape_pairs_512():
    import hertz_cases as HC
    from peclet.dem import workloads as W
    return HC.shape_pairs(seed=32, n=64, L=10e-3, shell=W.hollow_cylinder_shell())


# (name, scene, calls, substeps per call, skin fraction); the shape cases drive the shape-pair
# forces (src/solver_hertz.hpp:454) with the analytic shell and the 512-point stratified shell
CASES = [("drum_spheres", _drum_spheres, 4, 10, 0.3), ("dense_drum", _dense_drum, 3, 20, 0.2),
         ("shape_pairs", _shape_pairs, 3, 10, 0.3), ("shape_pairs_512", _shape_pairs_512, 2, 10, 0.3)]


@pytest.mark.parametrize("precision,rtol", [("fp32", 0.0), ("fp64", 1e-12)])
@pytest.mark.parametrize("name,mk,calls,substeps,skin", CASES, ids=[c[0] for c in CASES])
def test_hertz_vs_oracle(gpu_api, orc_api, name, mk, calls, substeps, skin, precision, rtol):
    sc, extra = mk()
    a = P.build(gpu_api, sc, extra, precision)
    b = P.build(orc_api, sc, extra, precision)
    for k in range(calls):
        a.step_hertz(2e-6, substeps, skin)
        b.step_hertz(2e-6, substeps, skin)
        sa, sb = P.snapshot(a, products=False), P.snapshot(b, products=False)
        ka, xa = a.debug_hertz()
        kb, xb = b.debug_hertz()
        sa.update(hk=ka, hx=xa)
        sb.update(hk=kb, hx=xb)
        bad = P.diff(sa, sb, rtol=rtol)
        assert not bad, f"{name} {precision}: hertz call {k}: {bad[:4]}"


@pytest.mark.parametrize("precision,rtol", [("fp32", 0.0), ("fp64", 1e-12)])
def test_hertz_after_a_periodic_step(gpu_api, orc_api, precision, rtol):
    """Both engines keep their candidate pairs in one list. A periodic XPBD step between two Hertz calls
    leaves pairs with its ghost slots (numbers above the bodies') there, which the second call takes as it
    finds them: forces on the bodies, none on the ghosts."""
    sc = S.polydisperse_periodic()

    def extra(s):
        s.set_hertz_material(0, 1e7, 0.3)
        s.enable_periodicity(False, False, False)
    sc.planes = []
    a, b = P.build(gpu_api, sc, extra, precision), P.build(orc_api, sc, extra, precision)
    for s in (a, b):
        s.step_hertz(2e-6, 4, 0.3)
        s.enable_periodicity(True, True, False)
        s.step(1e-6)
        s.enable_periodicity(False, False, False)
        pairs = s.debug_pairs()
        assert pairs.max() >= sc.n
        s.step_hertz(2e-6, 3, 0.3)
    bad = P.diff(P.snapshot(a, products=False), P.snapshot(b, products=False), rtol=rtol)
    assert not bad, bad[:4]


@pytest.mark.parametrize("precision,rtol", [("fp32", 0.0), ("fp64", 1e-12)])
def test_failed_rebuild_keeps_the_engine_usable(gpu_api, orc_api, precision, rtol):
    """A pair-list rebuild whose allocation fails (refused by a test hook) leaves no list behind: the next
    call rebuilds it first and carries the histories over. The oracle's single call of 16 + 16 substeps, whose
    rebuild falls between them, is the reference."""
    sc, extra = _drum_spheres()
    a, b = P.build(gpu_api, sc, extra, precision), P.build(orc_api, sc, extra, precision)
    for s in (a, b):
        s.step_hertz(2e-6, 8, 0.005)
    b.step_hertz(2e-6, 32, 0.005)
    gpu_api.fn["debug_refuse_alloc"](1)
    try:
        with pytest.raises(Exception, match="refused"):
            a.step_hertz(2e-6, 32, 0.005)
    finally:
        gpu_api.fn["debug_refuse_alloc"](0)
    assert len(a.debug_hertz()[0]) == 0
    a.step_hertz(2e-6, 16, 0.005)
    sa, sb = P.snapshot(a, products=False), P.snapshot(b, products=False)
    (sa["hk"], sa["hx"]), (sb["hk"], sb["hx"]) = a.debug_hertz(), b.debug_hertz()
    bad = P.diff(sa, sb, rtol=rtol)
    assert not bad, bad[:4]


def _grains(touching, radius=1e-3):
    """Two large grains, the first and the last body, each covered by `touching` small ones."""
    k = np.arange(touching) + 0.5
    phi, theta = np.arccos(1 - 2 * k / touching), np.pi * (1 + 5 ** 0.5) * k
    u = np.stack([np.cos(theta) * np.sin(phi), np.sin(theta) * np.sin(phi), np.cos(phi)], 1)
    rho = max(1.5, (touching * 4.6 / (4 * np.pi)) ** 0.5 - 1)
    reach, r = (rho + 2.1) * radius, np.full(2 * touching + 2, radius)
    c = np.array([[reach, reach, reach], [3 * reach, reach, reach]])
    r[0] = r[-1] = rho * radius
    pos = np.concatenate([c[:1], c[0] + u * (rho + 0.99) * radius, c[1] + u * (rho + 0.99) * radius, c[1:]])
    im, inertia = W.sphere_props(r, 2500.0)
    rng = np.random.default_rng(touching)
    return W.Scene(name="grains", pos=pos, vel=rng.uniform(-0.1, 0.1, pos.shape), inv_mass=im,
                   inv_inertia=np.repeat(np.asarray(inertia)[:, None], 3, 1), scales=r / radius, global_scale=radius,
                   domain=((0, 0, 0), (4 * reach, 2 * reach, 2 * reach), (False,) * 3), material=(0.6, 0.0, 0.4),
                   dt=2e-6)


@pytest.mark.parametrize("precision,rtol", [("fp32", 0.0), ("fp64", 1e-12)])
@pytest.mark.parametrize("touching", [1, 8, 9, 16, 17, 32, 33, 257, 700])
def test_grains_of_many_contacts(gpu_api, orc_api, touching, precision, rtol):
    """A body's touching pairs are summed in pair order: in registers, by repeated minimum or by its block,
    at the edges of each (and of the block's stage of 256)."""
    sc = _grains(touching)
    a, b = (P.build(api, sc, lambda s: s.set_hertz_material(0, 1e7, 0.3), precision) for api in (gpu_api, orc_api))
    for _ in range(2):
        a.step_hertz(2e-6, 4, 0.3)
        b.step_hertz(2e-6, 4, 0.3)
    assert (np.abs(b.debug_hertz()[1]).sum(1) > 0).sum() >= 2 * touching
    sa, sb = P.snapshot(a, products=False), P.snapshot(b, products=False)
    (sa["hk"], sa["hx"]), (sb["hk"], sb["hx"]) = a.debug_hertz(), b.debug_hertz()
    bad = P.diff(sa, sb, rtol=rtol)
    assert not bad, bad[:4]


@pytest.mark.parametrize("precision,rtol", [("fp32", 0.0), ("fp64", 1e-12)])
def test_long_pair_lists(gpu_api, orc_api, precision, rtol):
    """From 100,000 pairs a thread tests four of a tile: a jittered lattice of 27,000 spheres whose list is above
    that (the other tests' lists are below), with a ragged last tile."""
    n, a = 30, 2.02e-3
    rng = np.random.default_rng(6)
    g = np.stack(np.meshgrid(*[np.arange(n)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = (g + 0.5) * a + rng.uniform(-3e-5, 3e-5, (n ** 3, 3))
    im, inertia = W.sphere_props(1e-3, 2500.0)
    sc = W.Scene(name="lattice", pos=pos, vel=rng.uniform(-0.2, 0.2, pos.shape), inv_mass=np.full(n ** 3, im),
                 inv_inertia=np.full((n ** 3, 3), inertia), global_scale=1e-3,
                 domain=((0, 0, 0), (n * a,) * 3, (False,) * 3), material=(0.6, 0.0, 0.4), dt=2e-6)
    x, y = (P.build(api, sc, lambda s: s.set_hertz_material(0, 1e7, 0.3), precision) for api in (gpu_api, orc_api))
    for _ in range(2):
        x.step_hertz(2e-6, 3, 1.0)
        y.step_hertz(2e-6, 3, 1.0)
    sx, sy = P.snapshot(x, products=False), P.snapshot(y, products=False)
    (sx["hk"], sx["hx"]), (sy["hk"], sy["hx"]) = x.debug_hertz(), y.debug_hertz()
    assert len(sy["hk"]) >= 100000 and len(sy["hk"]) % 1024
    bad = P.diff(sx, sy, rtol=rtol)
    assert not bad, bad[:4]


def test_hertz_rejects_periodic(gpu_api):
    """The reference refuses the Hertz engine on periodic domains (src/sim.hpp:629-634); the B200
    step raises the same error type."""
    sc = S.polydisperse_periodic()
    sim = P.build(gpu_api, sc, lambda s: s.set_hertz_material(0, 1e7, 0.3), "fp64")
    with pytest.raises(RuntimeError):
        sim.step_hertz(2e-6, 2, 0.3)
