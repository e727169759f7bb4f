"""Rollout gradients on every launch that tapes the forward: tile mode, the
cooperative grid, one cluster, one CTA.  The forward is the same bits on all of
them, so are its tape and the reverse sweep (whose launch shape is the cloth's
own): gradients are compared for equality."""
import numpy as np
import pytest

import numi_cloth as nc
from helpers import PLAIN, make_solver, small_square

pytestmark = pytest.mark.gpu

COLOURS = {"NUMI_CLOTH_TILES": "0"}
ONE_CTA = {"NUMI_CLOTH_GRID": "1"}


def _scene(side, contact, **kw):
    """A cloth with one corner on a grip, on the ground or in the air; with
    `contact` spheres fall onto it within the rollout."""
    scene = small_square(side=side, fruits=6 if contact else 0, gripCorners=1, stretchCompliance=1e-4,
                         shearCompliance=2e-4, bendCompliance=1e-3, **kw)
    if contact:
        scene.fruits["velocityAndGroundImpulse"][:, 2] = -1.0
    return scene


def _rollout(scene, substeps=24):
    cfg = nc.substep_configs(scene, substeps)
    cfg["gripTargetAndActive"][:, 2] -= np.linspace(0.0, 0.004, substeps, dtype=np.float32)
    rng = np.random.default_rng(scene.n)
    tracked = np.sort(rng.choice(scene.n, 16, replace=False)).astype(np.uint32)
    x = scene.particles["positionAndInverseMass"][tracked, :3].astype(np.float64)
    return cfg, tracked, x + rng.normal(0.0, 2e-3, (substeps // 12, 16, 3))


def _run(scene, sched, env=None, settle=0, every=8, repeats=1):
    cfg, tracked, targets = _rollout(scene)
    sv = make_solver(scene, env=env)
    sv.snapshot(0)
    for _ in range(settle):   # a small cloth takes tile mode once it has stepped
        sv.step(nc.substep_configs(scene, 48), sched)
    for _ in range(repeats):
        sv.restore(0)
        r = sv.rollout_grad(cfg, sched, tracked, targets, 12, checkpoint_every=every)
    out = dict(r, particles=sv.particles(), info=sv.launch_info(), failure=sv.failure())
    sv.close()
    return out


def _same_gradients(a, b):
    assert a["failure"] == 0 and b["failure"] == 0
    assert np.array_equal(a["particles"], b["particles"])
    assert a["nonsmooth"] == b["nonsmooth"]
    for name in ("loss", "grads", "damping", "grip"):
        assert np.array_equal(a[name], b[name]), name


@pytest.mark.parametrize("contact", [False, True], ids=["free", "contact"])
@pytest.mark.parametrize("sweeps", [0, 1, 2])
def test_tile_mode_tape_of_a_small_cloth(contact, sweeps):
    """A cloth that has stepped enough for its tile plan against the same on
    its cluster; with contact the friction sweep moves velocities while the
    tiles begin the next substep."""
    sched = nc.Schedule.make(**dict(PLAIN, strainSweeps=sweeps, damping=0.5))
    scene = _scene(40, contact)
    tiled = _run(scene, sched, settle=4)
    plain = _run(scene, sched, env=COLOURS, settle=4)
    assert tiled["info"]["last_tiles"] and not plain["info"]["last_tiles"]
    assert (tiled["nonsmooth"] > 0) == contact
    _same_gradients(tiled, plain)


@pytest.mark.parametrize("contact", [False, True], ids=["free", "contact"])
def test_tape_of_a_large_cloth(contact):
    """Above 4,096 particles: tile mode, colour by colour on the cooperative
    grid, and one CTA."""
    sched = nc.Schedule.make(**dict(PLAIN, damping=0.5))
    scene = _scene(72, contact)
    tiled = _run(scene, sched)
    plain = _run(scene, sched, env=COLOURS)
    one = _run(scene, sched, env=ONE_CTA)
    assert tiled["info"]["last_tiles"] and tiled["info"]["grid"] > 1
    assert not plain["info"]["last_tiles"] and plain["info"]["grid"] > 1
    assert one["info"]["grid"] == 1
    _same_gradients(tiled, plain)
    _same_gradients(tiled, one)


def _regrab(scene, substeps=24):
    """The grip lets go half way and takes hold again elsewhere (a later
    generation); the second loss' targets are what the rollout reaches, so
    only the first, before the re-grab, has gradients."""
    cfg, tracked, targets = _rollout(scene, substeps)
    half = substeps // 2
    cfg["gripControl"][half:, 0] += 1
    cfg["gripTargetAndActive"][half:, 0] += np.float32(0.003)
    cfg["gripTargetAndActive"][half:half + 2, 3] = 0.0   # open for two substeps
    sched = nc.Schedule.make(**dict(PLAIN, damping=0.5))
    sv = nc.ClothSolver(scene)
    sv.step(cfg, sched)
    x = sv.particles()["positionAndInverseMass"][tracked, :3].astype(np.float64)
    assert sv.failure() == 0 and int(sv.grips()["particle"][0, 1]) == int(cfg["gripControl"][-1, 0])
    sv.close()
    return cfg, sched, tracked, np.stack([targets[0], x])


@pytest.mark.parametrize("every", [5, 12, 24])
@pytest.mark.parametrize("side", [12, 40, 72], ids=["one-cta", "cluster", "tiles"])
def test_gradients_before_a_regrab(side, every):
    """The reverse sweep meets every substep's own grips, not the last
    generation's: gradients up to a re-grab are those of the rollout that
    ends there (sums in other segments: 1e-10)."""
    scene = _scene(side, False)
    cfg, sched, tracked, targets = _regrab(scene)
    sv = nc.ClothSolver(scene)
    sv.snapshot(0)
    half = sv.rollout_grad(cfg[:12], sched, tracked, targets[:1], 12, checkpoint_every=12)
    sv.restore(0)
    full = sv.rollout_grad(cfg, sched, tracked, targets, 12, checkpoint_every=every)
    sv.close()
    batched = []
    for c, t in ((cfg[:12], targets[:1]), (cfg, targets)):
        solvers = [nc.ClothSolver(scene) for _ in range(2)]
        batch = nc.ClothBatch(solvers)
        r = batch.rollout_grad(np.stack([c, c]), sched, tracked, np.stack([t, t]), 12, checkpoint_every=every)
        batched.append((r["loss"][1], r["grads"][1], r["damping"][1]))
        batch.close()
    assert np.abs(half["grip"]).max() > 0.0 and half["loss"] > 0.0
    scale = np.abs(half["grip"]).max()
    assert np.allclose(full["grip"][:12], half["grip"], rtol=1e-10, atol=1e-10 * scale)
    assert np.array_equal(full["grip"][12:], np.zeros((12, 6)))
    for a, b in ((full, half),):
        assert np.allclose(a["loss"], b["loss"], rtol=1e-12)
        assert np.allclose(a["grads"], b["grads"], rtol=1e-10, atol=1e-10 * np.abs(b["grads"]).max())
        assert np.allclose(a["damping"], b["damping"], rtol=1e-10)
    for a, b in zip(batched[1], (half["loss"], half["grads"], half["damping"])):
        assert np.allclose(a, b, rtol=1e-10, atol=1e-10 * np.abs(b).max())


def _tape_limit(monkeypatch, scene, substeps):
    """Limits the tape to about `substeps` substeps (at least one interval is
    always taped)."""
    phases = 2 * len(np.unique(scene.distances["particlesAndColor"][:, 2])) + 12
    monkeypatch.setenv("NUMI_CLOTH_TAPE_BYTES", str(int(substeps * phases * scene.n * 16)))


@pytest.mark.parametrize("side, spheres", [(9, 0), (40, 0), (40, 2), (72, 0)])
@pytest.mark.parametrize("every", [1, 5, 8, 24])
def test_equal_bits_however_the_rollout_is_taped(monkeypatch, side, spheres, every):
    """The whole rollout on one tape, in segments of several intervals or of
    one: the same bits (spheres far above, which never touch)."""
    scene = small_square(side=side, fruits=spheres, gripCorners=1, stretchCompliance=1e-4, shearCompliance=2e-4,
                         bendCompliance=1e-3, fruitHeightMin=2.0, fruitHeightMax=3.0)
    sched = nc.Schedule.make(**dict(PLAIN, damping=0.5))
    whole = _run(scene, sched, every=every)
    for substeps in (1, 13):
        _tape_limit(monkeypatch, scene, substeps)
        _same_gradients(_run(scene, sched, every=every), whole)
    monkeypatch.delenv("NUMI_CLOTH_TAPE_BYTES")
    _same_gradients(_run(scene, sched, every=every, repeats=3), whole)


@pytest.mark.parametrize("every", [5, 24])
def test_equal_bits_however_a_batch_is_taped(monkeypatch, every):
    scenes = [_scene(side, False) for side in (12, 33, 40)]
    sched = nc.Schedule.make(**dict(PLAIN, damping=0.5))
    cfg, tracked, targets = _rollout(scenes[0])
    out = []
    for limit in (None, 1, 13):
        if limit is not None:
            _tape_limit(monkeypatch, scenes[2], 1.7 * limit)
        solvers = [nc.ClothSolver(s) for s in scenes]
        batch = nc.ClothBatch(solvers)
        cfgs = np.stack([_rollout(s)[0] for s in scenes])
        r = batch.rollout_grad(cfgs, sched, tracked, np.stack([targets] * 3), 12, checkpoint_every=every)
        out.append((r["loss"], np.concatenate(r["grads"]), r["damping"], r["nonsmooth"],
                    *[sv.particles() for sv in solvers]))
        batch.close()
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)


def test_equal_bits_after_a_rollout_with_contact():
    """What a handle's earlier rollout met changes no bit of the next."""
    scene = _scene(24, True)
    free = scene.fruits.copy()
    free["positionAndInverseMass"][:, 2] += 5.0
    free["previousAndRadius"][:, 2] += 5.0
    sched = nc.Schedule.make(**dict(PLAIN, damping=0.5))
    cfg, tracked, targets = _rollout(scene)
    sv = nc.ClothSolver(scene)
    sv.snapshot(0)
    runs = []
    for fruits in (scene.fruits, free, free, scene.fruits, free):
        sv.restore(0)
        sv.write_fruits(fruits)
        runs.append(sv.rollout_grad(cfg, sched, tracked, targets, 12, checkpoint_every=8))
    assert [r["nonsmooth"] > 0 for r in runs] == [True, False, False, True, False]
    for a, b in ((0, 3), (1, 2), (1, 4)):
        for name in ("loss", "grads", "damping", "grip"):
            assert np.array_equal(runs[a][name], runs[b][name]), (a, b, name)
