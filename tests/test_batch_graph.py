"""A captured batch step replays its own launch whatever the batch stepped in
between: another kernel family (its descriptors have another residency and
barrier), another number of substeps (its Configs lie elsewhere)."""
import numpy as np
import pytest

import numi_cloth as nc
from helpers import PLAIN, lift_trajectory_path, small_square

pytestmark = pytest.mark.gpu

EDGES = dict(PLAIN, primitiveSelf=1)


def _cloths(sides):
    scenes = [small_square(side=side, fruits=2, seed=side) for side in sides]
    return scenes, [nc.ClothSolver(s) for s in scenes]


def _configs(scenes, first, count):
    return np.stack([nc.substep_configs(s, first + count)[first:] for s in scenes])


# two cloths: a cluster each without the family; eighty: one CTA each, a
# larger residency without the family than with it
@pytest.mark.parametrize("sides", [(40, 24), (72, 40) + (9,) * 78], ids=["clusters", "one-cta"])
@pytest.mark.parametrize("captured, between, substeps", [(PLAIN, EDGES, 4), (EDGES, PLAIN, 4), (PLAIN, PLAIN, 7),
                                                         (PLAIN, EDGES, 3)],
                         ids=["plain-edges", "edges-plain", "more-substeps", "edges-fewer-substeps"])
def test_replay_after_another_launch(sides, captured, between, substeps):
    import torch
    scenes, solvers = _cloths(sides)
    _, ref = _cloths(sides)
    captured, between = nc.Schedule.make(**captured), nc.Schedule.make(**between)
    cfg, other = _configs(scenes, 0, 4), _configs(scenes, 4, substeps)
    plain = nc.ClothBatch(ref)
    for c, s in ((cfg, captured), (other, between), (cfg, captured), (other, between), (cfg, captured)):
        plain.step(c, s)
    batch = nc.ClothBatch(solvers)
    pinned = torch.empty(cfg.nbytes, dtype=torch.uint8, pin_memory=True)
    pinned.numpy()[:] = np.frombuffer(cfg.tobytes(), np.uint8)
    batch.capture(pinned, 4, captured)
    batch.replay()
    for _ in range(2):
        batch.step(other, between)
        batch.replay()
    for sv, rv in zip(solvers, ref):
        assert sv.failure() == 0 and rv.failure() == 0
        assert np.array_equal(sv.particles(), rv.particles())
        assert np.array_equal(sv.fruits(), rv.fruits())
    batch.close()
    plain.close()


@pytest.mark.parametrize("shape", [(0, 256), (0, 512), (1024, 256)], ids=["two-an-sm", "one-an-sm", "resident"])
def test_edge_family_on_bags_equals_alone(shape):
    """The produce bag's edge/edge contacts in a batch: the box tree's lists in
    global memory (two CTAs an SM, for whose bags' some 2,600 segments half an
    SM has no room) and in shared memory."""
    scene = nc.bag_scene(scenario="recorded", timestep=1.0 / 2880.0)
    motion = nc.GripTrajectory(lift_trajectory_path())
    cfg = motion.configs(scene.config, scene.handle_base, 0, 6, 1.0 / 2880.0)
    sched = nc.Schedule.make(**dict(EDGES, strainSweeps=3, finalPasses=2, selfCollision=1))
    alone = nc.ClothSolver(scene)
    alone.step(cfg, sched)
    assert alone.failure() == 0 and alone.edge_contacts()[0] > 0
    small = small_square(side=14, fruits=1)
    scenes = [scene, small, scene]
    solvers = [nc.ClothSolver(s) for s in scenes]
    batch = nc.ClothBatch(solvers)
    batch.set_shape(*shape)
    batch.step(np.stack([cfg, nc.substep_configs(small, 6), cfg]), sched)
    for k in (0, 2):
        assert solvers[k].failure() == 0 and solvers[k].edge_contacts() == alone.edge_contacts()
        assert np.array_equal(solvers[k].particles(), alone.particles())
    batch.close()
