"""The edge/edge family on a cooperative grid of more CTAs than SMs."""
import numpy as np
import pytest

import numi_cloth as nc
from helpers import bag_frame_configs, run_gpu

pytestmark = pytest.mark.gpu


def test_edge_grid_no_larger_than_its_tree_allows():
    """The box tree's shared memory leaves one CTA to an SM: the launch runs on
    as many as are co-resident, with the bits of any grid."""
    scene = nc.bag_scene(scenario="recorded", timestep=1.0 / 2880.0)
    cfg = bag_frame_configs(scene, 0, 4, 1.0 / 2880.0)
    sched = nc.Schedule.make(iterations=1, strainSweeps=3, reconcilePasses=2, finalPasses=2, certificatePasses=0,
                             earlyExit=1, selfCollision=1, aerodynamics=1, sweptGround=1, sweptFruitYarn=1, frictions=1,
                             primitiveSelf=1)
    wide = run_gpu(scene, cfg, sched, grid=200)
    default = run_gpu(scene, cfg, sched)
    assert 7 < wide["info"]["grid"] <= 200 and default["info"]["grid"] < 7
    assert wide["failure"] == 0 and default["failure"] == 0
    assert np.array_equal(wide["particles"], default["particles"])
