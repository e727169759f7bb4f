"""Tile plans of small cloths over a handle's life: built beside the stepping
thread, taken up without touching other streams, kept through material
changes (rewritten in place, on the handle's stream), given back with the
handle."""
import numpy as np
import pytest

import numi_cloth as nc
from helpers import PLAIN, make_solver, small_square

pytestmark = pytest.mark.gpu

COLOURS = {"NUMI_CLOTH_TILES": "0"}
SCHED = nc.Schedule.make(**dict(PLAIN, selfCollision=1))


def _scene(side=40):
    return small_square(side=side, fruits=3, gripCorners=1, stretchCompliance=1e-6, shearCompliance=2e-6,
                        bendCompliance=1e-4)


def _stepped(scene, env=None, stream=None):
    """A solver past the substeps after which a plan is taken up."""
    sv = make_solver(scene, env=env)
    if stream is not None:
        sv.set_stream(stream.cuda_stream)
    cfg = nc.substep_configs(scene, 48)
    for _ in range(4):
        sv.step(cfg, SCHED)
    return sv


def _changes(count):
    """Compliances of the stretch, shear and bend groups in turn."""
    rng = np.random.default_rng(3)
    now = {"distance": [np.float32(1e-6), np.float32(2e-6)], "bend": [np.float32(1e-4)]}
    for k in range(count):
        fam, at = (("distance", 0), ("bend", 0), ("distance", 1))[k % 3]
        to = np.float32(now[fam][at] * np.exp(rng.uniform(-0.3, 0.3)))
        yield fam, float(now[fam][at]), float(to)
        now[fam][at] = to


@pytest.mark.parametrize("side, env", [(40, {}), (96, {}), (120, {"NUMI_CLOTH_TILE_GRID": "5"})],
                         ids=["small", "large", "streamed"])
def test_material_changes_between_steps(side, env):
    scene = _scene(side)
    cfg = nc.substep_configs(scene, 6)
    tiled, plain = _stepped(scene, env), _stepped(scene, COLOURS)
    for fam, old, new in _changes(7):
        for sv in (tiled, plain):
            sv.replace_compliance(fam, old, new)
            sv.step(cfg, SCHED)
        assert tiled.launch_info()["last_tiles"] and not plain.launch_info()["last_tiles"]
        assert np.array_equal(tiled.particles(), plain.particles())
        assert np.array_equal(tiled.distances(), plain.distances())
    assert tiled.failure() == 0 and plain.failure() == 0


def test_material_changes_take_no_memory():
    import torch
    scene = _scene()
    cfg = nc.substep_configs(scene, 1)
    sv = _stepped(scene)
    sv.failure()
    free = torch.cuda.mem_get_info()[0]
    for fam, old, new in _changes(300):
        sv.replace_compliance(fam, old, new)
        sv.step(cfg, SCHED)
    assert sv.failure() == 0 and sv.launch_info()["last_tiles"]
    assert torch.cuda.mem_get_info()[0] == free


def test_material_change_and_step_in_a_capture():
    """A step captured after a material change, and the change itself."""
    import torch
    scene = _scene()
    cfg = nc.substep_configs(scene, 6)
    stream = torch.cuda.Stream()
    captured, plain = _stepped(scene, stream=stream), _stepped(scene, COLOURS)
    captured.replace_compliance("distance", 1e-6, 3e-6)
    captured.failure()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        captured.replace_compliance("bend", 1e-4, 2e-4)
        captured.step(cfg, SCHED)
    graph.replay()
    torch.cuda.synchronize()
    plain.replace_compliance("distance", 1e-6, 3e-6)
    plain.replace_compliance("bend", 1e-4, 2e-4)
    plain.step(cfg, SCHED)
    assert captured.failure() == 0
    assert np.array_equal(captured.particles(), plain.particles())


def test_plan_taken_up_during_another_streams_capture():
    """The launches that start a plan's build and take it up leave a capture
    of another stream on the same thread valid."""
    import torch
    scene = _scene()
    cfg = nc.substep_configs(scene, 16)
    mine, other = torch.cuda.Stream(), torch.cuda.Stream()
    sv = make_solver(scene)
    sv.set_stream(mine.cuda_stream)
    sv.step(cfg, SCHED)   # allocates its Configs and grid
    sv.failure()
    x = torch.zeros(4, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=other):
        for _ in range(9):
            sv.step(cfg, SCHED)
        x += 1.0
    graph.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 4.0
    assert sv.failure() == 0 and sv.launch_info()["last_tiles"]
    plain = make_solver(scene, env=COLOURS)
    for _ in range(10):
        plain.step(cfg, SCHED)
    assert np.array_equal(sv.particles(), plain.particles())


def test_handles_closed_while_their_plans_are_built():
    scene = _scene()
    cfg = nc.substep_configs(scene, 20)
    for rounds in (2, 3, 7):
        solvers = [nc.ClothSolver(scene) for _ in range(24)]
        for _ in range(rounds):
            for sv in solvers:
                sv.step(cfg, SCHED)
        for sv in solvers[::2]:
            sv.close()
        assert all(sv.failure() == 0 for sv in solvers[1::2])
        first = solvers[1].particles()
        assert all(np.array_equal(sv.particles(), first) for sv in solvers[3::2])
        for sv in solvers[1::2]:
            sv.close()


def test_per_cta_trace_of_a_small_cloth():
    """The per-CTA stamps stay available once a small cloth takes tile mode,
    one CTA more than its cluster."""
    scene = _scene()
    sv = make_solver(scene, env={"NUMI_CLOTH_TRACE": "48", "NUMI_CLOTH_TRACE_CTA": "1"})
    cfg = nc.substep_configs(scene, 48)
    for frame in range(4):
        sv.step(cfg, SCHED)
        t = sv.trace_cta(48)
        info = sv.launch_info()
        assert t.shape[2] == info["grid"] and sv.failure() == 0
        assert info["last_tiles"] == (frame >= 2)
        assert (t[:, 0, :] > 0).all() and (np.diff(t[:, 0, :].astype(np.int64), axis=0) > 0).all()


def test_plans_of_handles_on_several_threads():
    """Threads with handles and streams of their own, whose plans are built and
    taken up, materials changed and gradients taken side by side."""
    import threading

    import torch
    scene = _scene(30)
    cfg = nc.substep_configs(scene, 16)
    tracked = np.arange(4, dtype=np.uint32)
    target = scene.particles["positionAndInverseMass"][None, :4, :3].astype(np.float64) + 1e-3
    smooth = nc.Schedule.make(**dict(PLAIN, damping=0.5))
    out, errors = {}, []

    def work(name):
        try:
            stream = torch.cuda.Stream()
            solvers = [make_solver(scene) for _ in range(4)]
            for sv in solvers:
                sv.set_stream(stream.cuda_stream)
            for k in range(10):
                for sv in solvers:
                    sv.step(cfg, SCHED)
                if k == 8:
                    for sv in solvers:
                        sv.replace_compliance("distance", 1e-6, 3e-6)
            grads = [sv.rollout_grad(cfg, smooth, tracked, target, 16) for sv in solvers]
            out[name] = [(sv.failure(), sv.launch_info()["last_tiles"], sv.particles(), g["loss"], g["grads"])
                         for sv, g in zip(solvers, grads)]
            for sv in solvers:
                sv.close()
        except Exception as e:   # noqa: BLE001
            errors.append(e)

    work("alone")
    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    ref = out["alone"][0]
    assert ref[0] == 0 and ref[1]
    for rows in out.values():
        for failure, tiles, particles, loss, grads in rows:
            assert failure == 0 and tiles
            assert np.array_equal(particles, ref[2])
            assert loss == ref[3] and np.array_equal(grads, ref[4])
