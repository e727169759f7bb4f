"""Performance cases of the cloth solver: the calls that programs make.

Every case goes through the public Python entry points (ClothSolver,
ClothBatch, calibrate.Calibration).  Five kinds:

  step         one cloth, host records in, substeps, host records out: the
               contract of a host application that owns the state
  batch        many square cloths of uneven sizes: an episode from their
               start, one captured frame of all of them replayed frame by
               frame, every state read back at its end
  rollout      loss and reverse-mode gradients of one cloth's rollout
  rollouts     the same for many candidates in one call
  calibration  one evaluation of a fit of the produce bag's material

Inputs come from the seed alone.  exact() restates the contact-free cloth
(constraints, grips, strain limit, free-falling spheres) in float64 torch;
gradients come from its autograd.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.abspath("numi-solver_b200"))
import numi_cloth as nc  # noqa: E402
from numi_cloth import calibrate as cal  # noqa: E402

LIFT = os.path.join("tests", "golden", "lift-v1.csv")
DT = 1.0 / 2880.0
FRAME = 48   # substeps of a 60 Hz frame

# schedules: the square cloths' frame, the batch's (no self contact), the
# differentiable rollout's, the calibration's and the produce bag's
SQUARE = dict(iterations=1, strainSweeps=1, reconcilePasses=0, finalPasses=0, certificatePasses=0, earlyExit=0,
              aerodynamics=0, sweptGround=1, frictions=1, selfCollision=1)
BATCH = dict(SQUARE, selfCollision=0)
ROLLOUT = dict(BATCH, damping=0.5)
CALIBRATION = dict(BATCH, strainSweeps=3)
BAG = dict(iterations=1, strainSweeps=3, reconcilePasses=8, finalPasses=2, certificatePasses=128, earlyExit=1,
           selfCollision=1, aerodynamics=1, sweptGround=1, sweptFruitYarn=1, frictions=1, release=1)
SOFT = (1.0e-3, 2.0e-3, 1.0e-2)   # stretch, shear, bend compliance of the rollouts (m/N)
TRACKED, LOSS_EVERY = 32, 12


def listed():
    return [
        # an interactive control loop on a small cloth: one substep per call,
        # where the copies and launches count
        {"name": "substep_24", "kind": "step", "scene": "square", "side": 24, "spheres": 6, "height": 0.5,
         "drop": 0.05, "substeps": 1, "settle": 0},
        # a small cloth lying on the ground under spheres, one rendered frame
        # (particles resident on a cluster)
        {"name": "frame_61_resting", "kind": "step", "scene": "square", "side": 61, "spheres": 9, "height": 0.1,
         "drop": 0.05, "substeps": FRAME, "settle": 20},
        # an odd-sized cloth on the cooperative grid, spheres resting on it
        {"name": "frame_97_resting", "kind": "step", "scene": "square", "side": 97, "spheres": 33, "height": 0.1,
         "drop": 0.05, "substeps": FRAME, "settle": 20},
        # the 65,536-particle cloth with 64 spheres, before the spheres land
        {"name": "frame_256_falling", "kind": "step", "scene": "square", "side": 256, "spheres": 64, "height": 0.5,
         "drop": 0.05, "substeps": FRAME, "settle": 0},
        # the same cloth once it lies folded on the ground under the spheres
        {"name": "frame_256_resting", "kind": "step", "scene": "square", "side": 256, "spheres": 64, "height": 0.5,
         "drop": 0.05, "substeps": FRAME, "settle": 40},
        # the largest single cloth
        {"name": "frame_512_falling", "kind": "step", "scene": "square", "side": 512, "spheres": 64, "height": 0.5,
         "drop": 0.05, "substeps": FRAME, "settle": 0},
        # the produce bag on the recorded lift, the full reference schedule
        {"name": "bag_frame", "kind": "step", "scene": "bag", "edges": False, "substeps": FRAME, "settle": 2},
        # the same with the edge/edge yarn self-collision family
        {"name": "bag_frame_edges", "kind": "step", "scene": "bag", "edges": True, "substeps": FRAME, "settle": 2},
        # many cloths at once (training data, environments): short episodes
        {"name": "batch_192", "kind": "batch", "cloths": 192, "smallest": 16, "largest": 96, "substeps": FRAME,
         "frames": 4},
        # trajectory optimisation: one cloth's gradients
        {"name": "rollout_64", "kind": "rollout", "side": 64, "spheres": 4, "substeps": 96, "checkpoint": 8},
        # a population of candidates of the same rollout
        {"name": "rollouts_16", "kind": "rollouts", "side": 64, "spheres": 4, "substeps": 96, "checkpoint": 8,
         "candidates": 16},
        # material calibration of the produce bag
        {"name": "calibration_96", "kind": "calibration", "candidates": 96, "substeps": FRAME, "checkpoint": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "bag", "batch", "rollout", "rollouts", "calibration"])
    if kind == "step":
        side = _log(rng, 16, 400)
        resting = rng.random() < 0.5
        most = max(1, min(64, side * side // 160))
        return {"kind": "step", "scene": "square", "side": side, "spheres": rng.randint(1, most),
                "height": 0.1 if resting else rng.uniform(0.1, 0.5), "drop": 0.05,
                "substeps": _log(rng, 1, FRAME), "settle": rng.randint(15, 25) if resting else 0}
    if kind == "bag":
        return {"kind": "step", "scene": "bag", "edges": rng.random() < 0.5, "substeps": _log(rng, 8, FRAME),
                "settle": rng.randint(0, 4)}
    if kind == "batch":
        return {"kind": "batch", "cloths": _log(rng, 8, 192), "smallest": rng.randint(12, 24),
                "largest": rng.randint(32, 96), "substeps": _log(rng, 8, FRAME), "frames": rng.randint(1, 4)}
    if kind == "calibration":
        return {"kind": "calibration", "candidates": _log(rng, 8, 96), "substeps": 12 * rng.randint(1, 4),
                "checkpoint": rng.choice([4, 6, 8])}
    case = {"kind": kind, "side": rng.randint(20, 64), "spheres": rng.randint(0, 4), "substeps": 12 * rng.randint(1, 8),
            "checkpoint": rng.choice([4, 6, 8])}
    if kind == "rollouts":
        case["candidates"] = _log(rng, 4, 16)
    return case


# ------------------------------------------------------------- inputs -----

def _square_step_scene(case, seed):
    """A square cloth held by two corners, spheres above it, with small
    seeded velocities."""
    side = case["side"]
    most = 0.05 if side > 48 else 0.02
    scene = nc.square_scene(side=side, height=case["height"], fruitCount=case["spheres"], seed=7919 * seed + 11,
                            fruitRadiusMin=min(0.02, 0.5 * most), fruitRadiusMax=most,
                            fruitHeightMin=case["height"] + case["drop"], fruitHeightMax=case["height"] + 0.5,
                            timestep=DT)
    rng = np.random.default_rng([seed, side])
    scene.particles["velocity"][:, :3] = rng.normal(0.0, 0.01, (scene.n, 3)).astype(np.float32)
    return scene


def _rollout_scene(case, compliance):
    """A square cloth with a 3 x 3 corner patch on compliant grips."""
    side = case["side"]
    scene = nc.square_scene(side=side, spacing=0.004, height=0.12, gripCorners=1, fruitCount=case["spheres"],
                            fruitRadiusMin=0.01, fruitRadiusMax=0.03, fruitHeightMin=0.15, fruitHeightMax=0.25,
                            stretchCompliance=compliance[0], shearCompliance=compliance[1],
                            bendCompliance=compliance[2], timestep=DT, seed=20260310)
    corner = scene.grips[0]
    pos = scene.particles["positionAndInverseMass"][:, :3].astype(np.float64)
    ids = [i * side + j for i in range(3) for j in range(3)]
    grips = np.zeros(len(ids), scene.grips.dtype)
    for g, i in enumerate(ids):
        off = pos[i] - pos[0]
        grips[g]["particle"] = (i, corner["particle"][1], 0, 0)
        grips[g]["targetOffsetAndCompliance"] = (off[0], off[1], off[2], corner["targetOffsetAndCompliance"][3])
    scene.grips = grips
    scene.config["control"][0, 3] = len(grips)
    return scene


def _rollout_configs(scene, substeps, rng):
    """The grip moves at most 3 cm, outwards and down, and turns at most 8
    degrees, from rest (pushed inwards, a flat cloth buckles to a side that
    rounding picks)."""
    cfg = nc.substep_configs(scene, substeps)
    s = np.arange(1, substeps + 1) / substeps
    ramp = 0.5 - 0.5 * np.cos(np.pi * s)
    direction = -np.abs(rng.normal(size=3))
    direction /= np.linalg.norm(direction)
    trans = direction[None, :] * (rng.uniform(0.01, 0.03) * substeps / 96.0 * ramp)[:, None]
    axis = rng.normal(size=3)
    axis /= np.linalg.norm(axis)
    half = 0.5 * np.radians(rng.uniform(2.0, 8.0)) * substeps / 96.0 * ramp
    cfg["gripTargetAndActive"][:, :3] = (cfg["gripTargetAndActive"][:, :3] + trans).astype(np.float32)
    cfg["gripOrientation"] = np.concatenate([axis[None, :] * np.sin(half)[:, None], np.cos(half)[:, None]],
                                            axis=1).astype(np.float32)
    return cfg


def _rollout_inputs(case, seed):
    """Scenes (one per candidate, compliances around SOFT), the grip's
    motion, tracked particles and targets a few millimetres off the start."""
    rng = np.random.default_rng([seed, case["side"], 3])
    count = case.get("candidates", 1)
    shift = np.exp(rng.normal(0.0, 0.3, (count, 3)))
    scenes = [_rollout_scene(case, [c * f for c, f in zip(SOFT, row)]) for row in shift]
    cfg = _rollout_configs(scenes[0], case["substeps"], rng)
    tracked = np.sort(rng.choice(scenes[0].n, TRACKED, replace=False)).astype(np.uint32)
    start = scenes[0].particles["positionAndInverseMass"][tracked, :3].astype(np.float64)
    targets = start + rng.normal(0.0, 0.003, (count, case["substeps"] // LOSS_EVERY, TRACKED, 3))
    return scenes, cfg, tracked, targets


def _pinned(like):
    buf = torch.empty(like.nbytes, dtype=torch.uint8, pin_memory=True).numpy().view(like.dtype).reshape(like.shape)
    buf[:] = like
    return buf


def prepare(case, seed):
    torch.zeros(1, device="cuda")
    return globals()["_prepare_" + case["kind"]](case, seed)


def _prepare_step(case, seed):
    count, settle = case["substeps"], case["settle"]
    if case["scene"] == "bag":
        # the material differs from seed to seed within the calibrated range
        m = nc.material_defaults()
        rng = np.random.default_rng([seed, 5])
        for name in ("axialBodyComplianceMPerN", "knotCompliance", "bendBodyComplianceMPerN"):
            setattr(m, name, getattr(m, name) * float(np.exp(rng.uniform(-0.2, 0.2))))
        scene = nc.bag_scene(material=m, scenario="recorded", timestep=DT)
        motion = nc.GripTrajectory(LIFT)
        cfgs = [motion.configs(scene.config, scene.handle_base, f * FRAME, FRAME, DT) for f in range(settle + 1)]
        sched = nc.Schedule.make(**dict(BAG, primitiveSelf=int(case["edges"])))
    else:
        scene = _square_step_scene(case, seed)
        cfgs = [nc.substep_configs(scene, FRAME)] * (settle + 1)
        sched = nc.Schedule.make(**SQUARE)
    solver = nc.ClothSolver(scene)
    for f in range(settle):
        solver.step(cfgs[f], sched)
    particles, fruits = _pinned(solver.particles()), _pinned(solver.fruits())
    return {"kind": "step", "solver": solver, "sched": sched, "cfg": _pinned(cfgs[settle][:count]),
            "particles": particles, "fruits": fruits, "out_particles": _pinned(particles),
            "out_fruits": _pinned(fruits)}


def _batch_sides(case):
    return np.random.default_rng([case["cloths"], case["smallest"], case["largest"]]).integers(
        case["smallest"], case["largest"] + 1, case["cloths"])


def _batch_scenes(case, seed):
    rng = np.random.default_rng([seed, 17])
    # the sizes are the case's, the materials and the spheres' places the seed's
    sides = _batch_sides(case)
    out = []
    for k, side in enumerate(sides):
        c = np.exp(rng.uniform(np.log(1e-9), np.log(1e-4), 3))
        scene = nc.square_scene(side=int(side), spacing=0.005, height=0.2, gripCorners=0, stretchCompliance=float(c[0]),
                                shearCompliance=float(c[1]), bendCompliance=float(c[2]),
                                fruitCount=1 + k % 4, fruitRadiusMin=0.01, fruitRadiusMax=0.03,
                                fruitHeightMin=0.2015, fruitHeightMax=0.4, seed=1000 * seed + k, timestep=DT)
        # the spheres move down onto the cloth at up to 1 m/s
        scene.fruits["velocityAndGroundImpulse"][:, 2] = -rng.uniform(0.2, 1.0, len(scene.fruits)).astype(np.float32)
        out.append((scene, float(rng.uniform(0.0, 0.05))))
    return out


def _prepare_batch(case, seed):
    solvers, cfgs = [], []
    stream = torch.cuda.Stream()   # a captured graph cannot use the default stream
    for scene, damping in _batch_scenes(case, seed):
        sv = nc.ClothSolver(scene)
        sv.set_stream(stream.cuda_stream)
        sv.set_damping(damping)
        sv.snapshot(0)
        solvers.append(sv)
        cfgs.append(nc.substep_configs(scene, case["substeps"]))
    cfg = np.stack(cfgs)
    pinned = torch.empty(cfg.nbytes, dtype=torch.uint8, pin_memory=True)
    pinned.numpy()[:] = np.frombuffer(cfg.tobytes(), np.uint8)
    batch = nc.ClothBatch(solvers)
    batch.set_stream(stream.cuda_stream)
    batch.capture(pinned, case["substeps"], nc.Schedule.make(**BATCH))
    sizes = [sv.n for sv in solvers]
    rows = _pinned(np.zeros(sum(sizes), nc.abi.PARTICLE))
    frows = _pinned(np.zeros(sum(len(sv.scene.fruits) for sv in solvers), nc.abi.FRUIT))
    return {"kind": "batch", "solvers": solvers, "batch": batch, "stream": stream, "pinned": pinned,
            "frames": case["frames"], "out_particles": rows, "out_fruits": frows}


def _prepare_rollout(case, seed):
    scenes, cfg, tracked, targets = _rollout_inputs(case, seed)
    solver = nc.ClothSolver(scenes[0])
    solver.snapshot(0)
    return {"kind": "rollout", "solver": solver, "cfg": cfg, "sched": nc.Schedule.make(**ROLLOUT), "tracked": tracked,
            "targets": targets[0], "checkpoint": case["checkpoint"], "out": _pinned(scenes[0].particles)}


def _prepare_rollouts(case, seed):
    scenes, cfg, tracked, targets = _rollout_inputs(case, seed)
    solvers = [nc.ClothSolver(s) for s in scenes]
    for sv in solvers:
        sv.snapshot(0)
    return {"kind": "rollouts", "solvers": solvers, "batch": nc.ClothBatch(solvers),
            "cfg": np.stack([cfg] * len(solvers)), "sched": nc.Schedule.make(**ROLLOUT), "tracked": tracked,
            "targets": targets, "checkpoint": case["checkpoint"],
            "out": _pinned(np.stack([s.particles for s in scenes]))}


def _prepare_calibration(case, seed):
    rng = np.random.default_rng([seed, 23])
    scene = nc.bag_scene(scenario="recorded", timestep=DT)
    cfg = nc.GripTrajectory(LIFT).configs(scene.config, scene.handle_base, 0, case["substeps"], DT)
    m = nc.material_defaults()
    base = np.array([getattr(m, name) for _, name in cal.BAG_PARAMS], np.float32)
    z = scene.particles["positionAndInverseMass"][:, 2]
    tracked = np.unique(np.concatenate([scene.cuff[:48:2][:20], np.argsort(z)[:20]])).astype(np.uint32)
    start = scene.particles["positionAndInverseMass"][tracked, :3].astype(np.float64)
    targets = start + rng.normal(0.0, 0.002, (case["substeps"] // LOSS_EVERY, len(tracked), 3))
    n = case["candidates"]
    logc = np.log(base.astype(np.float64))[None, :] + rng.uniform(-1.0, 1.0, (n, len(base)))
    fit = cal.Calibration([scene] * n, cfg, nc.Schedule.make(**CALIBRATION), tracked, targets, LOSS_EVERY, base,
                          checkpoint_every=case["checkpoint"])
    # an optimiser moves the parameters between evaluations
    return {"kind": "calibration", "fit": fit, "logc": [logc, logc + rng.normal(0.0, 0.05, logc.shape)],
            "damping": rng.uniform(0.0, 0.05, n), "turn": 0}


# ---------------------------------------------------------------- run -----

def _particle_rows(p):
    return p.view(np.float32).reshape(len(p), 12)


def _fruit_rows(f):
    return f.view(np.float32).reshape(len(f), 24)[:, :20]   # the identity words stay out


def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_step(st):
    sv = st["solver"]
    sv.write_particles(st["particles"])
    sv.write_fruits(st["fruits"])
    sv.step(st["cfg"], st["sched"])
    sv.particles(out=st["out_particles"])
    sv.fruits(out=st["out_fruits"])
    return {"particles": _particle_rows(st["out_particles"]), "fruits": _fruit_rows(st["out_fruits"]),
            "failure": sv.failure()}


def _run_batch(st):
    for sv in st["solvers"]:
        sv.restore(0)
    for _ in range(st["frames"]):
        st["batch"].replay()
    at = fat = 0
    failure = 0
    for sv in st["solvers"]:
        f = len(sv.scene.fruits)
        sv.particles(out=st["out_particles"][at:at + sv.n])
        sv.fruits(out=st["out_fruits"][fat:fat + f])
        at, fat = at + sv.n, fat + f
        failure |= sv.failure()
    return {"particles": _particle_rows(st["out_particles"]), "fruits": _fruit_rows(st["out_fruits"]),
            "failure": failure}


def _run_rollout(st):
    st["solver"].restore(0)
    r = st["solver"].rollout_grad(st["cfg"], st["sched"], st["tracked"], st["targets"], LOSS_EVERY,
                                  checkpoint_every=st["checkpoint"])
    return {"loss": r["loss"], "grads": r["grads"], "damping": r["damping"], "grip": r["grip"],
            "nonsmooth": r["nonsmooth"], "particles": _particle_rows(st["solver"].particles(out=st["out"]))}


def _run_rollouts(st):
    for sv in st["solvers"]:
        sv.restore(0)
    r = st["batch"].rollout_grad(st["cfg"], st["sched"], st["tracked"], st["targets"], LOSS_EVERY,
                                 checkpoint_every=st["checkpoint"])
    for sv, rows in zip(st["solvers"], st["out"]):
        sv.particles(out=rows)
    return {"loss": r["loss"], "grads": np.stack(r["grads"]), "damping": r["damping"],
            "nonsmooth": r["nonsmooth"].astype(np.int64),
            "particles": st["out"].view(np.float32).reshape(*st["out"].shape, 12)}


def _run_calibration(st):
    st["turn"] ^= 1
    loss, grads, damping, rough = st["fit"].evaluate(st["logc"][st["turn"]], st["damping"])
    return {"loss": loss, "grads": grads, "damping": damping, "nonsmooth": rough.astype(np.int64)}


# --------------------------------------------------------------- work -----

def _counts(scene):
    d = len(scene.distances)
    limited = int((scene.distances["material"][:, 3] > 0).sum())
    return scene.n, d, len(scene.knots), len(scene.bends), limited, len(scene.fruits)


def _work_of(counts, substeps, sweeps, passes, self_contact):
    """State in and out and every record once; the arithmetic of the
    projections (square roots and quotients as one operation each)."""
    n, d, k, b, limited, f = counts
    nbytes = 2 * (48 * n + 96 * f) + 28 * d + 24 * k + 24 * b + 224 * substeps
    per = 60 * n + 35 * d + 110 * k + 60 * b + 20 * limited * sweeps + 12 * limited * passes * (f > 0)
    per += (100 * n if self_contact else 0) + f * f * 5 + 200 * f
    return np.array([nbytes, per * substeps], np.float64)


def work(case):
    kind, substeps = case["kind"], case["substeps"]
    if kind == "step" and case["scene"] == "bag":
        w = _work_of(_counts(nc.bag_scene()), substeps, 3, 3, True)
    elif kind == "step":
        side = case["side"]
        w = _work_of((side * side, 2 * side * (side - 1) + 2 * (side - 1) ** 2, 0, 2 * side * (side - 2),
                      2 * side * (side - 1), case["spheres"]), substeps, 1, 1, True)
    elif kind == "batch":
        w = sum(_work_of((s * s, 2 * s * (s - 1) + 2 * (s - 1) ** 2, 0, 2 * s * (s - 2), 2 * s * (s - 1), 2),
                         substeps * case["frames"], 1, 1, False) for s in (int(v) for v in _batch_sides(case)))
    elif kind == "calibration":
        # forward, its replay, and two to three times the forward for the
        # reverse sweep; the state comes in once and the gradients go out
        w = case["candidates"] * np.array([0.5, 4.0]) * _work_of(_counts(nc.bag_scene()), substeps, 3, 1, False)
    else:
        side = case["side"]
        w = _work_of((side * side, 2 * side * (side - 1) + 2 * (side - 1) ** 2, 0, 2 * side * (side - 2),
                      2 * side * (side - 1), case["spheres"]), substeps, 1, 1, False)
        w = case.get("candidates", 1) * np.array([0.5, 4.0]) * w
    return {"bytes": float(w[0]), "flops": float(w[1])}


# -------------------------------------------------------------- exact -----

def exact(case, seed):
    """Float64 values where the cloth meets nothing: the first frames of the
    square cloths and the rollouts.  Contact on the ground, under spheres
    and in the bag is a long sequence of order-dependent decisions with no
    value apart from that order."""
    if case["kind"] == "step" and case["scene"] == "square" and case["settle"] == 0:
        if case["side"] ** 2 * case["substeps"] > 110000 * FRAME:
            return None   # the float64 cloth would take too long
        return _exact_step(case, seed)
    if case["kind"] in ("rollout", "rollouts"):
        return _exact_rollout(case, seed)
    return None


def _runs(colours):
    edges = np.flatnonzero(np.diff(colours)) + 1
    return list(zip(np.concatenate([[0], edges]), np.concatenate([edges, [len(colours)]])))


def _rotate(q, v):
    """v turned by the unit quaternion q (xyzw)."""
    u = torch.cross(q[:3].expand_as(v), v, dim=-1) * 2.0
    return v + q[3] * u + torch.cross(q[:3].expand_as(u), u, dim=-1)


class _Cloth:
    """A square cloth in float64, [candidates, particles, 3], one XPBD
    iteration and one strain sweep per substep in the colour order of the
    records."""

    def __init__(self, scenes):
        s = scenes[0]
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a, np.float64))  # noqa: E731
        ids = lambda a: torch.from_numpy(a.astype(np.int64))                 # noqa: E731
        self.x0 = t(np.stack([c.particles["positionAndInverseMass"][:, :3] for c in scenes]))
        self.v0 = t(np.stack([c.particles["velocity"][:, :3] for c in scenes]))
        self.w = t(s.particles["positionAndInverseMass"][:, 3])
        d, b = s.distances, s.bends
        self.d_runs = [slice(int(lo), int(hi)) for lo, hi in _runs(d["particlesAndColor"][:, 2])]
        self.b_runs = [slice(int(lo), int(hi)) for lo, hi in _runs(b["particlesAndColor"][:, 3])]
        self.d_ij = ids(d["particlesAndColor"][:, :2])
        self.b_ij = ids(b["particlesAndColor"][:, [0, 2]])
        self.d_rest, self.d_limit = t(d["material"][:, 0]), t(d["material"][:, 3])
        self.b_rest = t(b["material"][:, 0])
        self.d_c = t(np.stack([c.distances["material"][:, 1] for c in scenes]))
        self.b_c = t(np.stack([c.bends["material"][:, 2] for c in scenes]))
        self.g_id = ids(s.grips["particle"][:, 0])
        self.g_off = t(s.grips["targetOffsetAndCompliance"][:, :3])
        self.g_c = t(s.grips["targetOffsetAndCompliance"][:, 3])

    def _pull(self, x, ij, rest, alpha):
        i, j = ij[:, 0], ij[:, 1]
        diff = x[:, j] - x[:, i]
        length = diff.square().sum(-1, keepdim=True).sqrt()
        wi, wj = self.w[i, None], self.w[j, None]
        push = diff * ((rest[:, None] - length) / ((wi + wj + alpha[..., None]) * length))
        return x.index_add(1, i, -push * wi).index_add(1, j, push * wj)

    def _limit(self, x, ij, rest, limit):
        i, j = ij[:, 0], ij[:, 1]
        diff = x[:, j] - x[:, i]
        length = diff.square().sum(-1, keepdim=True).sqrt()
        over = (length - (rest * (1.0 + limit))[:, None]).clamp(min=0.0)
        wi, wj = self.w[i, None], self.w[j, None]
        pull = diff * (over / ((wi + wj) * length))
        return x.index_add(1, i, pull * wi).index_add(1, j, -pull * wj)

    def substep(self, x, v, cfg, damping, scale=None, pose=None):
        """(positions, velocities) after one substep; scale: factors of the
        stretch, shear, bend and grip compliances [4, candidates, 1]; pose:
        shift and turn of the grip [6]."""
        dt = float(cfg["gravityAndTimestep"][3])
        g = torch.from_numpy(cfg["gravityAndTimestep"][:3].astype(np.float64))
        one = 1.0 if scale is None else None   # no factors
        prev = x
        x = x + (v + g * dt) * (1.0 / (1.0 + damping * dt)) * dt
        for r in self.d_runs:
            shear = self.d_limit[r] <= 0.0
            f = one if one else torch.where(shear, scale[1], scale[0])
            x = self._pull(x, self.d_ij[r], self.d_rest[r], self.d_c[:, r] * f / dt ** 2)
        for r in self.b_runs:
            x = self._pull(x, self.b_ij[r], self.b_rest[r], self.b_c[:, r] * (one or scale[2]) / dt ** 2)
        target = torch.from_numpy(cfg["gripTargetAndActive"][:3].astype(np.float64))
        arm = _rotate(torch.from_numpy(cfg["gripOrientation"].astype(np.float64)), self.g_off)
        goal = target + arm
        if pose is not None:
            goal = goal + pose[:3] + torch.cross(pose[3:].expand_as(arm), arm, dim=-1)
        at = x[:, self.g_id]
        alpha = self.g_c * (one or scale[3]) / dt ** 2
        wg = self.w[self.g_id]
        x = x.index_add(1, self.g_id, (goal - at) * (wg / (wg + alpha))[..., None])
        for r in self.d_runs:
            on = self.d_limit[r] > 0.0
            if bool(on.any()):
                x = self._limit(x, self.d_ij[r][on], self.d_rest[r][on], self.d_limit[r][on])
        return x, (x - prev) / dt, prev


def _exact_step(case, seed):
    scene = _square_step_scene(case, seed)
    cloth = _Cloth([scene])
    x, v = cloth.x0, cloth.v0
    with torch.no_grad():
        for cfg in nc.substep_configs(scene, case["substeps"]):
            x, v, prev = cloth.substep(x, v, cfg, 0.0)
    rows = _particle_rows(scene.particles).astype(np.float64)
    rows[:, 0:3], rows[:, 4:7], rows[:, 8:11], rows[:, 11] = x[0].numpy(), prev[0].numpy(), v[0].numpy(), 0.0
    falling = _fruit_rows(scene.fruits).astype(np.float64)
    dt = float(cfg["gravityAndTimestep"][3])
    for _ in range(case["substeps"]):
        falling[:, 8:11] += cfg["gravityAndTimestep"][:3].astype(np.float64) * dt
        falling[:, 4:7] = falling[:, 0:3]
        falling[:, 0:3] += falling[:, 8:11] * dt
    return {"particles": rows, "fruits": falling, "failure": None}


def _exact_rollout(case, seed):
    scenes, cfg, tracked, targets = _rollout_inputs(case, seed)
    cloth = _Cloth(scenes)
    count = len(scenes)
    theta = torch.zeros(4, count, 1, dtype=torch.float64, requires_grad=True)
    damping = torch.full((count, 1, 1), float(np.float32(ROLLOUT["damping"])), dtype=torch.float64,
                         requires_grad=True)
    pose = torch.zeros(len(cfg), 6, dtype=torch.float64, requires_grad=True)
    x, v = cloth.x0, cloth.v0
    at = torch.from_numpy(tracked.astype(np.int64))
    goal = torch.from_numpy(targets)
    loss = torch.zeros(count, dtype=torch.float64)
    for s, c in enumerate(cfg):
        x, v, prev = cloth.substep(x, v, c, damping, torch.exp(theta), pose[s])
        if (s + 1) % LOSS_EVERY == 0:
            loss = loss + (x[:, at] - goal[:, s // LOSS_EVERY]).square().sum((1, 2))
    loss.sum().backward()
    # the groups' order: each family's compliances ascending
    order = [0, 1, 2, 3]
    grads = []
    for k, scene in enumerate(scenes):
        c = np.unique(scene.distances["material"][:, 1])
        stretch = scene.distances["material"][scene.distances["material"][:, 3] > 0, 1][0]
        o = order if stretch == c[0] else [1, 0, 2, 3]
        grads.append(theta.grad[o, k, 0].numpy())
    rows = np.stack([_particle_rows(scene.particles) for scene in scenes]).astype(np.float64)
    for at, value in ((0, x), (4, prev), (8, v)):
        rows[:, :, at:at + 3] = value.detach().numpy()
    rows[:, :, 11] = 0.0
    out = {"particles": rows, "loss": loss.detach().numpy(), "grads": np.stack(grads), "damping": damping.grad[:, 0, 0].numpy(),
           "nonsmooth": None}
    if case["kind"] == "rollout":
        out = {"particles": rows[0], "loss": float(loss[0].detach()), "grads": grads[0], "damping": np.float64(out["damping"][0]),
               "grip": pose.grad.numpy(), "nonsmooth": None}
    return out
