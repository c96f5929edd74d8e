"""Performance cases of the rigid-body step: what a program that uses this
package asks of it, from one game world to the largest batches, in both
arithmetic forms, with the learned warm start and its training.

A case is a dict of plain values, told apart by "kind":

  frames   step a batch from a saved state and read the bodies back: a game's
           frame, an episode, a batch of simulations (WorldBatch.step)
  calls    one frame through the separate calls, with the caller's own test
           order (integrate, collide, resolve)
  host     a program that holds its bodies on the host: upload, integrate,
           download
  train    one epoch of the warm-start network

Every pass of a simulation starts from the same state (cz_restore, or the
uploaded arrays), so passes on one state do the same work; a training pass goes
on from the last one's parameters.
"""
import math

import numpy as np
import torch

from cubez_gb300 import learned, scenes
from cubez_gb300.batch import FORM_FP32, FORM_FP64, WorldBatch

DT = 1.0 / 60.0
# the dynamic state: what a program reads after stepping
STATE = ("position", "orientation", "velocity", "rotation")


def _frames(name, scene, worlds, bodies, form, settle, frames, warm=False):
    return {"name": name, "kind": "frames", "scene": scene, "worlds": worlds, "bodies": bodies, "form": form,
            "settle": settle, "frames": frames, "warm": warm}


def listed():
    return [
        # one frame of a game's single world of cubes and its poses: latency
        _frames("game_frame", "cubedrop", 1, 20, "fp64", 120, 1),
        # the example's own workload: 20 cubes dropped, 240 frames in one call
        _frames("game_episode", "cubedrop", 1, 20, "fp64", 0, 240),
        # one frame by separate calls in the ballistic example's test order,
        # with a static body and sleeping bodies (the Go API's way of stepping)
        {"name": "caller_order", "kind": "calls", "bodies": 26, "form": "fp64", "settle": 60},
        # a few worlds of many sizes (8 to 64 bodies): too few to fill the GPU
        _frames("few_worlds", "mixed", 61, 0, "fp32", 150, 30),
        # colliders with Offsets, an odd number of worlds
        _frames("offsets", "offsets", 1001, 24, "fp64", 120, 20),
        # the batched float64 workload: 4096 worlds of 8 to 64 bodies
        _frames("batched_fp64", "mixed", 4096, 0, "fp64", 120, 30),
        # the precision workload at full size, from landing to rest
        _frames("precision_fp32", "precision", 16384, 32, "fp32", 120, 60),
        # the same scenes with the learned warm start
        _frames("learned_fp32", "precision", 8192, 32, "fp32", 120, 30, warm=True),
        # dense piles of 1024 cubes
        _frames("piles_fp32", "piles", 64, 1024, "fp32", 40, 8),
        # a few piles of an odd size, float64
        _frames("piles_fp64", "piles", 5, 252, "fp64", 40, 8),
        # bodies held on the host: up, one Integrate, down
        {"name": "host_state", "kind": "host", "worlds": 4096, "bodies": 0, "form": "fp32"},
        # one epoch of the warm-start network at the default mini-batch
        {"name": "train_epoch", "kind": "train", "rows": 262147, "batch": 8192},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# body-frames of one pass that a drawn case may ask for, by form: a fraction of
# the largest listed case
_MOST = {"fp32": 16384 * 32 * 60, "fp64": 4096 * 36 * 30}


def _unnamed(case):
    return {k: v for k, v in case.items() if k != "name"}


def draw(rng):
    kind = rng.choice(["mixed", "mixed", "precision", "precision", "offsets", "cubedrop", "piles", "warm", "calls",
                       "host", "train"])
    form = rng.choice(["fp32", "fp64"])
    if kind == "train":
        return {"kind": "train", "rows": _log_int(rng, 3000, 262147), "batch": _log_int(rng, 1000, 8192)}
    if kind == "calls":
        return {"kind": "calls", "bodies": rng.randint(3, 40), "form": form, "settle": rng.randint(40, 80)}
    if kind == "host":
        return {"kind": "host", "worlds": _log_int(rng, 1, 4096), "bodies": 0, "form": form}
    if kind == "cubedrop":
        frames = _log_int(rng, 1, 200)
        return _unnamed(_frames("", "cubedrop", 1, 20, form, rng.randint(0, 240), frames))
    if kind == "piles":
        # lattices of 4 layers; above 64 bodies the large-world resolver runs
        side = rng.randint(4, 12)
        worlds = _log_int(rng, 1, 48)
        return _unnamed(_frames("", "piles", worlds, 4 * side * (side + rng.randint(0, 1)), form, rng.randint(20, 50),
                                rng.randint(2, 6)))
    warm = kind == "warm"
    scene = "precision" if warm else kind
    form = "fp32" if warm else form
    bodies = 0 if scene == "mixed" else rng.randint(2, 31) * 2 + (0 if scene == "precision" else rng.randint(0, 1))
    worlds = _log_int(rng, 1, 16384 if form == "fp32" else 4096)
    per_frame = worlds * (bodies or 36)
    frames = max(1, min(_log_int(rng, 1, 60), _MOST[form] // per_frame))
    return _unnamed(_frames("", scene, worlds, bodies, form, rng.randint(30, 200), frames, warm=warm))


def _lattice(bodies):
    """(nx, nz) of a 4-layer lattice of `bodies` cubes, as near a square as it divides."""
    per = bodies // 4
    nx = max(d for d in range(1, int(math.isqrt(per)) + 1) if per % d == 0)
    return nx, per // nx


def _scene(name, worlds, bodies, seed):
    if name == "cubedrop":
        return scenes.cubedrop(seed=seed)
    if name == "mixed":
        # worlds of 8 to 64 bodies, the same sizes for every seed: the first
        # bodies of worlds of 64
        counts = np.random.default_rng(worlds).integers(8, 65, worlds).astype(np.int32)
        full = scenes.mixed(num_worlds=worlds, seed=seed, min_bodies=64, max_bodies=64)
        keep = (np.arange(64)[None, :] < counts[:, None]).reshape(-1)
        return scenes.Scene(counts, full.plane, name=name, **{k: getattr(full, k)[keep] for k in scenes.Scene.FIELDS})
    if name == "precision":
        return scenes.precision(num_worlds=worlds, bodies=bodies, seed=seed)
    if name == "offsets":
        return scenes.offsets(num_worlds=worlds, bodies=bodies, seed=seed)
    nx, nz = _lattice(bodies)
    return scenes.piles(num_worlds=worlds, seed=seed, nx=nx, nz=nz, ny=4)


def _form(case):
    return FORM_FP32 if case["form"] == "fp32" else FORM_FP64


# (offset, outputs, inputs) of the network's weight matrices
_WEIGHTS = ((learned.OFF_W1, learned.H, learned.IN), (learned.OFF_W2, learned.H, learned.H),
            (learned.OFF_W3, learned.H, learned.H), (learned.OFF_W4, learned.OUT, learned.H))


def _network(seed):
    """Parameters that predict about what a trained network does: a share of
    the impulse that would resolve each contact alone (feature 13), carried
    through the three layers by one unit each, beside small seeded weights."""
    rng = np.random.default_rng(seed)
    blob = np.zeros(learned.BLOB, np.float32)
    blob[learned.OFF_IS:learned.OFF_IS + learned.IN] = 1.0
    blob[learned.OFF_OS:learned.OFF_OS + learned.OUT] = 1.0
    for off, rows, cols in _WEIGHTS:
        w = rng.normal(0.0, 0.01 / math.sqrt(cols), (rows, cols)).astype(np.float32)
        w[0, 13 if off == learned.OFF_W1 else 0] = 0.7 if off == learned.OFF_W4 else 1.0
        blob[off:off + rows * cols] = w.reshape(-1)
    return blob


def _training_set(rows, seed):
    """Features and impulses with the shape of harvested ones: flags, counts,
    velocities of resting and of falling contacts, mostly positive normal
    impulses that the features explain in part."""
    rng = np.random.default_rng(seed)
    x = rng.normal(0.0, 1.0, (rows, learned.IN)).astype(np.float32)
    x *= np.linspace(0.2, 3.0, learned.IN, dtype=np.float32)
    x[:, 0] = 0.0
    x[:, 1] = 1.0
    x[:, 13] = np.abs(x[:, 13])
    x[:, 14] = rng.integers(1, 9, rows)
    x[:, 15] = 0.0
    x[:, 16:] = np.abs(x[:, 16:])
    w = rng.normal(0.0, 0.3, (learned.IN, learned.OUT)).astype(np.float32)
    y = np.tanh(x @ w)
    y[:, 0] = 0.6 * x[:, 13] + np.abs(y[:, 0])
    return x, y.astype(np.float32)


def _untrained(x, y, seed):
    """Initial parameters: uniform weights of variance 2 / inputs, zero biases,
    the data's feature mean and deviation and output scale."""
    rng = np.random.default_rng(seed + 1)
    blob = np.zeros(learned.BLOB, np.float32)
    for off, rows, cols in _WEIGHTS:
        bound = math.sqrt(6.0 / cols)
        blob[off:off + rows * cols] = rng.uniform(-bound, bound, rows * cols)
    blob[learned.OFF_MU:learned.OFF_IS] = x.mean(axis=0, dtype=np.float64)
    deviation = x.std(axis=0, dtype=np.float64)
    blob[learned.OFF_IS:learned.OFF_OS] = np.where(deviation < 1e-10, 0.0, 1.0 / (deviation + 1e-12))
    blob[learned.OFF_OS:] = np.sqrt((y.astype(np.float64) ** 2).mean(axis=0))
    return blob


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        x, y = _training_set(case["rows"], seed)
        t = learned.Trainer(seed=seed)
        t.set_data(x, y, normalize=False)
        t.set_params(_untrained(x, y, seed))
        return {"kind": kind, "trainer": t, "batch": case["batch"], "seed": seed}
    if kind == "host":
        scene = _scene("mixed", case["worlds"], 0, seed)
        batch = WorldBatch(scene.counts, form=_form(case), plane=scene.plane)
        return {"kind": kind, "batch": batch, "scene": scene}
    if kind == "calls":
        bodies = case["bodies"]
        scene = scenes.ballistic(num_worlds=1, bullets=bodies - 2, seed=seed)
        units = scenes.ballistic_units(bodies)
        batch = WorldBatch.from_scene(scene, form=_form(case), iteration_multiplier=8)
        for _ in range(case["settle"]):
            batch.integrate(DT)
            batch.collide(0, units)
            batch.resolve(DT)
        batch.snapshot()
        return {"kind": kind, "batch": batch, "units": units}
    scene = _scene(case["scene"], case["worlds"], case["bodies"], seed)
    batch = WorldBatch.from_scene(scene, form=_form(case))
    if case["warm"]:
        learned.set_warm_start(batch, _network(seed))
    frames = case["frames"]
    calls = max(1, case["settle"] // frames)  # at least one: it captures the rollout
    if case["settle"] < frames:
        batch.snapshot()
    for _ in range(calls):
        batch.step(frames, DT)
    if case["settle"] >= frames:
        batch.snapshot()
    return {"kind": kind, "batch": batch, "frames": frames}


def run(state):
    kind = state["kind"]
    if kind == "train":
        t = state["trainer"]
        losses = t.train(epochs=1, batch=state["batch"], lr=1e-3, seed=state["seed"])
        return {"losses": losses, "params": t.params()}
    batch = state["batch"]
    if kind == "host":
        batch.upload(state["scene"])
        batch.integrate(DT)
        return batch.download()
    batch.restore()
    if kind == "calls":
        batch.integrate(DT)
        batch.collide(0, state["units"])
        batch.resolve(DT)
    else:
        batch.step(state["frames"], DT)
    return batch.download(STATE)


def _bodies_of(case):
    if case["kind"] == "frames" or case["kind"] == "host":
        # worlds of 8 to 64 bodies hold 36 on average
        return case["worlds"] * (case["bodies"] or 36)
    return case["bodies"]


def work(case):
    if case["kind"] == "train":
        # rows in, parameters in and out; forward 9.4k multiply-adds a row,
        # backward twice that
        rows = case["rows"]
        return {"bytes": 4.0 * (rows * (learned.IN + learned.OUT) + 2 * learned.NPARAM), "flops": 2.0 * 3 * 9400 * rows}
    n = _bodies_of(case)
    real = 4 if case["form"] == "fp32" else 8
    if case["kind"] == "host":
        # host arrays in (position .. motion, 41 doubles and flags), the
        # downloaded state out (27 doubles and the awake flag); Integrate
        return {"bytes": n * (41 * 8.0 + 6 + 27 * 8 + 1), "flops": 250.0 * n}
    # bodies in (state, shape, mass and inertia: 36 reals), the state out as
    # doubles; per body and frame about 2200 operations: 250 of Integrate,
    # 1000 of the pair tests past the culls, 1000 of about 4 resolver
    # iterations (20 iterations in a dense pile)
    frames = case.get("frames", 1)
    ops = 6000.0 if case.get("scene") == "piles" else 2200.0
    return {"bytes": n * (36.0 * real + 13 * 8), "flops": ops * n * frames}


def _integrated(scene):
    """RigidBody.Integrate and CalculateDerivedData in 64 bits for bodies at
    the start of a scene (awake, no forces, CanSleep off)."""
    vel = (scene.velocity + scene.acceleration * DT) * (scene.linear_damping ** DT)[:, None]
    rot = scene.rotation * (scene.angular_damping ** DT)[:, None]
    pos = scene.position + vel * DT
    w, x, y, z = scene.orientation.T
    a, b, c = (rot * DT).T
    q = scene.orientation + 0.5 * np.stack([-a * x - b * y - c * z, a * w + b * z - c * y, b * w + c * x - a * z,
                                            c * w + a * y - b * x], axis=1)
    norm = np.sqrt((q * q).sum(axis=1))
    near = np.abs(1.0 - norm) < 1e-7 * (1.0 + norm)  # left as it is
    q = np.where(near[:, None], q, q / norm[:, None])
    w, x, y, z = q.T
    r = np.stack([1 - 2 * y * y - 2 * z * z, 2 * x * y - 2 * w * z, 2 * x * z + 2 * w * y,
                  2 * x * y + 2 * w * z, 1 - 2 * x * x - 2 * z * z, 2 * y * z - 2 * w * x,
                  2 * x * z - 2 * w * y, 2 * y * z + 2 * w * x, 1 - 2 * x * x - 2 * y * y], axis=1).reshape(-1, 3, 3)
    body = scene.inverse_inertia.reshape(-1, 3, 3).transpose(0, 2, 1)  # column-major
    world = r @ body @ r.transpose(0, 2, 1)
    return {"position": pos, "orientation": q, "velocity": vel, "rotation": rot,
            "inverse_inertia_world": np.ascontiguousarray(world.transpose(0, 2, 1)).reshape(-1, 9),
            "motion": scene.motion, "is_awake": scene.is_awake, "last_frame_acceleration": scene.acceleration}


def _mix(z):
    """The finaliser of the trainer's splitmix64 stream, on uint64 arrays."""
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _trained(case, seed):
    """One epoch of Adam in 64 bits, over the trainer's own shuffle."""
    rows, size = case["rows"], case["batch"]
    x, y = _training_set(rows, seed)
    blob = _untrained(x, y, seed).astype(np.float64)
    mu, inv = blob[learned.OFF_MU:learned.OFF_IS], blob[learned.OFF_IS:learned.OFF_OS]
    scale = blob[learned.OFF_OS:]
    order = list(range(rows))
    with np.errstate(over="ignore"):
        at = np.arange(rows - 1, 0, -1, dtype=np.uint64)
        drawn = _mix(np.uint64(seed) + np.arange(1, rows, dtype=np.uint64) * np.uint64(0x9E3779B97F4A7C15))
        for i, j in zip(at.tolist(), (drawn % (at + np.uint64(1))).tolist()):
            order[i], order[j] = order[j], order[i]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    xs = torch.from_numpy((x - mu) * inv).to(dev)
    ys = torch.from_numpy(y / scale).to(dev)
    order = torch.tensor(order, device=dev)
    shapes = ((learned.H, learned.IN), (learned.H,), (learned.H, learned.H), (learned.H,), (learned.H, learned.H),
              (learned.H,), (learned.OUT, learned.H), (learned.OUT,))
    p, off = [], 0
    for s in shapes:
        k = int(np.prod(s))
        p.append(torch.from_numpy(blob[off:off + k].reshape(s)).to(dev).requires_grad_(True))
        off += k
    m1 = [torch.zeros_like(q) for q in p]
    m2 = [torch.zeros_like(q) for q in p]
    total, step = 0.0, 0
    for b0 in range(0, rows, size):
        at = order[b0:b0 + size]
        h = xs[at]
        for k in (0, 2, 4):
            h = torch.relu(h @ p[k].T + p[k + 1])
        loss = ((h @ p[6].T + p[7] - ys[at]) ** 2).sum()
        total += float(loss.detach())
        step += 1
        for q, g, a, b in zip(p, torch.autograd.grad(loss / (learned.OUT * len(at)), p), m1, m2):
            a.mul_(0.9).add_(g, alpha=0.1)
            b.mul_(0.999).addcmul_(g, g, value=0.001)
            with torch.no_grad():
                q -= 1e-3 * (a / (1 - 0.9 ** step)) / ((b / (1 - 0.999 ** step)).sqrt() + 1e-8)
    blob[:learned.NPARAM] = torch.cat([q.detach().reshape(-1) for q in p]).cpu().numpy()
    return {"losses": np.array([total / (learned.OUT * rows)]), "params": blob}


def exact(case, seed):
    if case["kind"] == "host":
        return _integrated(_scene("mixed", case["worlds"], 0, seed))
    if case["kind"] == "train":
        return _trained(case, seed)
    # whole frames: a sequential solver of up to thousands of iterations a
    # world and frame, which plain numpy does not run in 20 seconds
    return None
