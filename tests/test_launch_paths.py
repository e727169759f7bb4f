"""Paths that a launch takes by the cloth's size and state, each against the
colour-by-colour launch, the cloth alone or the FP32 oracle (bit for bit), and
gradients across launch shapes (FP64 sums in another order: 1e-10, as the
batched gradients are held to)."""
import numpy as np
import pytest

import numi_cloth as nc
from helpers import PLAIN, gpu_fruit_positions, run_gpu, run_oracle, small_square

pytestmark = pytest.mark.gpu

SELF = dict(PLAIN, selfCollision=1)
ROLLOUT = dict(PLAIN, damping=0.5)
RESTING = dict(spacing=0.004, height=0.1, fruitRadiusMin=0.01, fruitRadiusMax=0.02, fruitHeightMin=0.1005,
               fruitHeightMax=0.14, timestep=1.0 / 2880.0)


def _same(a, b):
    assert a["failure"] == 0 and b["failure"] == 0
    for name in ("particles", "fruits"):
        assert np.array_equal(a[name], b[name]), name


def _spheres(count, pitch):
    """A small cloth far below `count` equal spheres on a grid of `pitch`
    (their diameter is 4 cm) with seeded offsets."""
    scene = nc.square_scene(side=12, fruitCount=count, height=0.1, fruitHeightMin=1.0, fruitHeightMax=5.0,
                            fruitRadiusMin=0.02, fruitRadiusMax=0.02, timestep=1.0 / 2880.0)
    rng = np.random.default_rng(count)
    k = np.arange(count)
    at = np.stack([k % 4, (k // 4) % 4, k // 16], axis=1) * pitch + rng.uniform(-1e-3, 1e-3, (count, 3))
    at[:, 2] += 0.5
    scene.fruits["positionAndInverseMass"][:, :3] = at.astype(np.float32)
    scene.fruits["previousAndRadius"][:, :3] = scene.fruits["positionAndInverseMass"][:, :3]
    return scene


@pytest.mark.parametrize("count, pitch", [(24, 0.0395), (25, 0.0395), (33, 0.0398), (64, 0.0398), (64, 0.03),
                                          (32, 0.02)],
                         ids=["walk", "fewest", "two-words", "most", "crowded", "far-moving"])
def test_sphere_pairs_equal_oracle(count, pitch):
    """Wavefronts of near pairs, and the walk where there are few colours,
    too many near pairs or motion beyond the proof."""
    scene = _spheres(count, pitch)
    cfg = nc.substep_configs(scene, 6)
    sched = nc.Schedule.make(**PLAIN)
    g = run_gpu(scene, cfg, sched)
    o = run_oracle(scene, cfg, sched)
    assert np.array_equal(gpu_fruit_positions(g).astype(np.float64), o["fruits"]["x"])
    assert np.array_equal(g["fruits"]["angularVelocity"][:, :3].astype(np.float64), o["fruits"]["omega"])


@pytest.mark.parametrize("side", [17, 31, 61])
def test_small_cloth_tiles_equal_cluster(side):
    """A small cloth's tile mode, taken up once it has stepped 128 substeps."""
    scene = nc.square_scene(side=side, fruitCount=min(9, side // 4), seed=side, **RESTING)
    cfg = nc.substep_configs(scene, 150)
    sched = nc.Schedule.make(**SELF)
    tiles = run_gpu(scene, cfg, sched, frames=5)
    plain = run_gpu(scene, cfg, sched, frames=5, env={"NUMI_CLOTH_TILES": "0"})
    assert tiles["info"]["last_tiles"] and not plain["info"]["last_tiles"]
    _same(tiles, plain)


@pytest.mark.parametrize("side, ctas", [(120, 5), (131, 7)])
def test_streamed_tile_items_equal_colour_by_colour(side, ctas):
    """Plans too large for shared memory: items streamed from global memory."""
    scene = nc.square_scene(side=side, fruitCount=12, seed=side, **RESTING)
    cfg = nc.substep_configs(scene, 12)
    sched = nc.Schedule.make(**SELF)
    tiles = run_gpu(scene, cfg, sched, env={"NUMI_CLOTH_TILE_GRID": str(ctas)})
    plain = run_gpu(scene, cfg, sched, env={"NUMI_CLOTH_TILES": "0"})
    assert tiles["info"]["last_tiles"] and tiles["info"]["grid"] == ctas
    _same(tiles, plain)


@pytest.mark.parametrize("sides", [(17,), (40, 64, 9), (110, 20), (64, 65, 96, 110) + (7,) * 72],
                         ids=["one", "clusters", "large-clusters", "one-cta"])
def test_fitted_batch_equals_alone(sides):
    """The default batch shape: a cluster per cloth, and one CTA per cloth with
    positions and velocities, positions alone (65 x 65 on) or nothing
    (110 x 110) in its shared memory."""
    scenes = [nc.square_scene(side=s, fruitCount=2, seed=s, **RESTING) for s in sides]
    cfg = np.stack([nc.substep_configs(s, 6) for s in scenes])
    sched = nc.Schedule.make(**PLAIN)
    solvers = [nc.ClothSolver(s) for s in scenes]
    batch = nc.ClothBatch(solvers)
    batch.step(cfg, sched)
    for sv, scene, c in list(zip(solvers, scenes, cfg))[:5]:
        alone = run_gpu(scene, c, sched)
        assert sv.failure() == 0 and alone["failure"] == 0
        assert np.array_equal(sv.particles(), alone["particles"])
        assert np.array_equal(sv.fruits(), alone["fruits"])
    batch.close()


def _rollout(scene, substeps):
    cfg = nc.substep_configs(scene, substeps)
    cfg["gripTargetAndActive"][:, 2] -= np.linspace(0.0, 0.004, substeps, dtype=np.float32)
    rng = np.random.default_rng(scene.n)
    tracked = np.sort(rng.choice(scene.n, 8, replace=False)).astype(np.uint32)
    x = scene.particles["positionAndInverseMass"][tracked, :3].astype(np.float64)
    return cfg, tracked, x + rng.normal(0.0, 2e-3, (substeps // 12, 8, 3))


@pytest.mark.parametrize("side, fruits", [(7, 0), (23, 2), (40, 0)])
def test_gradients_across_cluster_sizes(side, fruits):
    """One cloth's reverse sweep on its own cluster against the same cloth
    among 80 (one CTA each); fruits that touch nothing change nothing."""
    scene = small_square(side=side, fruits=fruits, gripCorners=1, stretchCompliance=1e-4, shearCompliance=2e-4,
                         bendCompliance=1e-3, height=0.0, groundEnabled=0, fruitHeightMin=0.3, fruitHeightMax=0.5)
    cfg, tracked, targets = _rollout(scene, 24)
    sched = nc.Schedule.make(**ROLLOUT)
    sv = nc.ClothSolver(scene)
    one = sv.rollout_grad(cfg, sched, tracked, targets, 12, checkpoint_every=7)
    ref = run_gpu(scene, cfg, sched)
    assert one["nonsmooth"] == 0 and np.array_equal(sv.particles(), ref["particles"])
    sv.close()
    solvers = [nc.ClothSolver(scene) for _ in range(80)]
    batch = nc.ClothBatch(solvers)
    r = batch.rollout_grad(np.stack([cfg] * 80), sched, tracked, np.stack([targets] * 80), 12, checkpoint_every=7)
    for k in (0, 41, 79):
        assert np.allclose(r["loss"][k], one["loss"], rtol=1e-12, atol=0.0)
        assert np.allclose(r["grads"][k], one["grads"], rtol=1e-10, atol=0.0)
        assert np.allclose(r["damping"][k], one["damping"], rtol=1e-10, atol=0.0)
    assert np.array_equal(solvers[79].particles(), ref["particles"])
    batch.close()


def test_gradients_with_fruit_contact_repeat():
    """A rollout that finds fruit contact after taping the forward gives the
    gradients of the one after it, which replays from the start."""
    scene = small_square(side=24, fruits=6, gripCorners=1, stretchCompliance=1e-4, shearCompliance=2e-4,
                         bendCompliance=1e-3)
    scene.fruits["velocityAndGroundImpulse"][:, 2] = -1.0   # onto the cloth within the rollout
    cfg, tracked, targets = _rollout(scene, 24)
    sched = nc.Schedule.make(**ROLLOUT)
    sv = nc.ClothSolver(scene)
    sv.snapshot(0)
    runs = []
    for _ in range(2):
        sv.restore(0)
        runs.append((sv.rollout_grad(cfg, sched, tracked, targets, 12, checkpoint_every=8), sv.particles()))
    assert runs[0][0]["nonsmooth"] > 0
    assert runs[0][0]["loss"] == runs[1][0]["loss"]
    for name in ("grads", "grip"):
        assert np.array_equal(runs[0][0][name], runs[1][0][name])
    assert np.array_equal(runs[0][1], runs[1][1])
    assert np.array_equal(runs[0][1], run_gpu(scene, cfg, sched)["particles"])


def test_compliance_groups_follow_replacements_and_restores():
    """The groups kept on the host: after values are replaced and merged, and
    after a restore brings old grip compliances back."""
    scene = small_square(side=9, fruits=0, gripCorners=2, stretchCompliance=1e-4, shearCompliance=2e-4,
                         bendCompliance=1e-3)
    sv = nc.ClothSolver(scene)
    stretch, shear, bend, grip = (np.float32(v) for v in (1e-4, 2e-4, 1e-3, 2e-4))
    sv.snapshot(0)
    assert sv.compliance_groups() == [("distance", float(stretch)), ("distance", float(shear)), ("bend", float(bend)),
                                      ("grip", float(grip))]
    sv.replace_compliance("distance", float(stretch), 5e-4)
    sv.replace_compliance("bend", float(bend), 2e-3)
    sv.replace_compliance("grip", float(grip), 7e-4)
    f = lambda v: float(np.float32(v))   # noqa: E731
    assert sv.compliance_groups() == [("distance", float(shear)), ("distance", f(5e-4)), ("bend", f(2e-3)),
                                      ("grip", f(7e-4))]
    sv.replace_compliance("distance", f(5e-4), float(shear))
    assert sv.compliance_groups() == [("distance", float(shear)), ("bend", f(2e-3)), ("grip", f(7e-4))]
    sv.restore(0)   # the grips are state, the constraints' materials are not
    assert sv.compliance_groups() == [("distance", float(shear)), ("bend", f(2e-3)), ("grip", float(grip))]
    fresh = nc.ClothSolver(scene)
    fresh.replace_compliance("distance", float(stretch), float(shear))
    fresh.replace_compliance("bend", float(bend), 2e-3)
    assert fresh.compliance_groups() == sv.compliance_groups()


@pytest.mark.parametrize("sides", [(17,), (40, 64, 9), (64, 65, 96, 110) + (7,) * 72], ids=["one", "clusters", "one-cta"])
def test_reported_batch_shape_is_accepted(sides):
    """A program that keeps the shape a batch or its tuner reported can set it
    again; chunks of no kind stay refused."""
    scenes = [nc.square_scene(side=s, fruitCount=2, seed=s, **RESTING) for s in sides]
    cfg = np.stack([nc.substep_configs(s, 4) for s in scenes])
    sched = nc.Schedule.make(**PLAIN)
    out = []
    for again in (False, True):
        solvers = [nc.ClothSolver(s) for s in scenes]
        batch = nc.ClothBatch(solvers)
        if again:
            for s in (batch.shape(), batch.tune(cfg, sched)):
                batch.set_shape(4096, 256)
                batch.set_shape(s["resident_chunk"], s["threads"])
                assert batch.shape()["threads"] == s["threads"]
            for bad in (3, 4097, 8192, max(s * s for s in sides) + 1):
                with pytest.raises(nc.ClothError):
                    batch.set_shape(bad, 512)
        batch.step(cfg, sched)
        out.append([sv.particles() for sv in solvers])
        batch.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_compliance_groups_after_captured_changes():
    """A captured change takes place when its graph is replayed, and a captured
    restore brings the grips' compliances back then."""
    import torch
    scene = small_square(side=9, fruits=0, gripCorners=2, stretchCompliance=1e-4, shearCompliance=2e-4,
                         bendCompliance=1e-3)
    stretch, shear, bend, grip = (float(np.float32(v)) for v in (1e-4, 2e-4, 1e-3, 2e-4))
    before = [("distance", stretch), ("distance", shear), ("bend", bend), ("grip", grip)]
    f = lambda v: float(np.float32(v))   # noqa: E731
    stream = torch.cuda.Stream()
    sv = nc.ClothSolver(scene)
    sv.set_stream(stream.cuda_stream)
    sv.snapshot(0)
    assert sv.compliance_groups() == before
    change, restore = torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()
    with torch.cuda.graph(change, stream=stream):
        sv.replace_compliance("bend", bend, 2e-3)
        sv.replace_compliance("grip", grip, 7e-4)
    with torch.cuda.graph(restore, stream=stream):
        sv.restore(0)
    assert sv.compliance_groups() == before
    change.replay()
    torch.cuda.synchronize()
    assert sv.compliance_groups() == before[:2] + [("bend", f(2e-3)), ("grip", f(7e-4))]
    restore.replay()
    torch.cuda.synchronize()
    assert sv.compliance_groups() == before[:2] + [("bend", f(2e-3)), ("grip", grip)]


@pytest.mark.parametrize("sides", [(40, 33, 24, 9) + (32,) * 300, (53, 40, 33, 24, 9) + (32,) * 300],
                         ids=["resident", "global"])
def test_fitted_batch_by_twos_equals_alone(sides):
    """More small cloths than SMs run two to an SM, on 256 threads each, with
    positions and velocities or positions alone (40 x 40) in half of its shared
    memory, or nothing where the largest does not fit (53 x 53); with the
    edge/edge family one to an SM.  (By ones they would take three turns.)"""
    scenes = {s: nc.square_scene(side=s, fruitCount=2, seed=s, **RESTING) for s in set(sides)}
    for extra in ({}, {"selfCollision": 1}, {"primitiveSelf": 1}):
        sched = nc.Schedule.make(**dict(PLAIN, **extra))
        solvers = [nc.ClothSolver(scenes[s]) for s in sides]
        batch = nc.ClothBatch(solvers)
        shape = batch.shape()
        assert shape["threads"] == 256 and shape["ctas"] > 148
        assert (shape["resident_chunk"] > 0) == (max(sides) <= 40)
        batch.set_shape(shape["resident_chunk"], shape["threads"])
        assert batch.shape() == shape
        cfg = np.stack([nc.substep_configs(scenes[s], 6) for s in sides])
        batch.step(cfg, sched)
        for k in (0, 1, 2, 3, 4, 5, len(sides) - 1):
            alone = run_gpu(scenes[sides[k]], cfg[k], sched)
            assert solvers[k].failure() == 0 and alone["failure"] == 0
            assert np.array_equal(solvers[k].particles(), alone["particles"]), (extra, k)
            assert np.array_equal(solvers[k].fruits(), alone["fruits"]), (extra, k)
        batch.close()
        for sv in solvers:
            sv.close()
