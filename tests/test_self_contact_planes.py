"""Point self contact of cloths in every axis plane: the grid's groups of
cells (2 x 2 x 2) are met at all parities, on both sides of the origin, and a
turned fold resolves as many pairs as a lying one."""
import numpy as np
import pytest

import numi_cloth as nc
from helpers import PLAIN, run_gpu, run_oracle
from test_gpu_parity import _check_bitexact

pytestmark = pytest.mark.gpu

SELF = dict(PLAIN, selfCollision=1)


def _fold(plane, shift, side=20):
    """Half of a cloth laid over the other half, 1.2 yarn radii above it and
    a fifth of a spacing off (one partner within the 2 mm each), in the plane normal to axis `plane`, moved by `shift`
    (in metres; the cells are 4 mm)."""
    scene = nc.square_scene(side=side, fruitCount=0, spacing=0.005, height=0.0, groundEnabled=0, gripCorners=0,
                            timestep=1.0 / 2880.0, seed=plane)
    p = scene.particles["positionAndInverseMass"][:, :3].astype(np.float64)
    i, j = np.divmod(np.arange(scene.n), side)
    over = i >= side // 2
    p[:, 0] = np.where(over, (side - 1 - i) + 0.2, i) * 0.005 - 0.03
    p[:, 1] = (j + 0.2 * over) * 0.005 - 0.05
    p[:, 2] = 0.0012 * over
    p = np.roll(p, plane - 2, axis=1) + shift
    for field in ("positionAndInverseMass", "previousAndMass"):
        scene.particles[field][:, :3] = p.astype(np.float32)
    return scene


@pytest.mark.parametrize("plane", [0, 1, 2], ids=["x", "y", "z"])
@pytest.mark.parametrize("shift", [0.0, 0.0041, -1.0027])
def test_fold_in_each_plane_equals_oracle(plane, shift):
    scene = _fold(plane, shift)
    cfg = nc.substep_configs(scene, 4)
    sched = nc.Schedule.make(**SELF)
    g = run_gpu(scene, cfg, sched)
    assert g["failure"] == 0 and g["self_contacts"][0] > 0
    _check_bitexact(g, run_oracle(scene, cfg, sched, bits=32))
