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
