"""A captured batch step replays its own launch whatever the batch stepped in
between: another kernel family (its descriptors have another residency and
barrier), another number of substeps (its Configs lie elsewhere)."""
import numpy as np
import pytest

import numi_cloth as nc
from helpers import PLAIN, small_square

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
