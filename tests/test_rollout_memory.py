"""Device memory of rollout gradients between calls: bounded over all handles
and batches of the process, given back with its owner and to an allocation
that finds no room."""
import numpy as np
import pytest

import numi_cloth as nc
from helpers import PLAIN, small_square

pytestmark = pytest.mark.gpu

SCHED = nc.Schedule.make(**dict(PLAIN, damping=0.5))


def _rollout(sv, scene, substeps):
    cfg = nc.substep_configs(scene, substeps)
    tracked = np.arange(4, dtype=np.uint32)
    x = scene.particles["positionAndInverseMass"][tracked, :3].astype(np.float64) + 1e-3
    return sv.rollout_grad(cfg, SCHED, tracked, np.tile(x, (1, 1, 1)), substeps, checkpoint_every=16)


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()


def test_kept_memory_is_bounded():
    """Rollouts of about 1.2 GB on sixteen handles, of which the process keeps
    a sixteenth of the device at most."""
    scene = small_square(side=72, fruits=0, gripCorners=1)
    solvers = [nc.ClothSolver(scene) for _ in range(16)]
    before, total = _free()
    ref = _rollout(solvers[0], scene, 512)
    assert before - _free()[0] > 1 << 29   # one is kept
    for sv in solvers[1:]:
        r = _rollout(sv, scene, 512)
        assert r["loss"] == ref["loss"] and np.array_equal(r["grads"], ref["grads"])
    assert before - _free()[0] <= total // 16 + (64 << 20)
    for sv in solvers:
        sv.close()
    assert before - _free()[0] <= 64 << 20


def test_kept_memory_goes_to_an_allocation_without_room():
    """A rollout whose checkpoint interval asks for more than the device has is
    refused as ever, after the idle workspaces are given back."""
    scene = small_square(side=72, fruits=0, gripCorners=1)
    sv, other = nc.ClothSolver(scene), nc.ClothSolver(scene)
    sv.snapshot(0)
    ref = _rollout(sv, scene, 256)
    held = _free()[0]
    substeps = 120000   # some 300 GB of tape in one interval
    cfg = nc.substep_configs(scene, substeps)
    x = np.zeros((1, 1, 3))
    with pytest.raises(nc.ClothError):
        other.rollout_grad(cfg, SCHED, np.array([0], np.uint32), x, substeps, checkpoint_every=substeps)
    assert _free()[0] - held > 1 << 28
    sv.restore(0)
    again = _rollout(sv, scene, 256)
    assert again["loss"] == ref["loss"] and np.array_equal(again["grads"], ref["grads"])
