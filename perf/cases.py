"""Performance cases: the calls a program makes through this package's public API.

Whole ticks.  A simulation is created once; a pass puts the scene back into its
saved state (device copies into `GpuPhysics.state_buffers()` on the handle's
own stream, as a rollout or a replay does) and steps it for a few ticks, whose
numbering starts over, so every pass is the same work.  It ends with the last
tick's readback, where a program looks at the error flags.  The results are
that tick's flags and counts and the body state (and, in the interactive
loop, the host snapshots).

Single operations on device tensors: the radix sort, the batched box
separating-axis test, and the learned parts' network (inference and training).
"""
import math

import numpy as np
import torch

from mechanic_b200 import abi, learned, ops, scenes
from mechanic_b200.net_init import init_params
from mechanic_b200.physics import GpuPhysics, GpuPhysicsConfig

TICK_KINDS = ("cubes", "grid", "dense", "chains", "batch", "loops")


def listed():
    return [
        # A small interactive scene: 1,000 falling cubes, every tick's snapshot read back to the
        # host before the next one (a game loop); launches and latency are what it pays for.
        {"name": "cubes_1k_loop", "kind": "cubes", "bodies": 1000, "warm": 30, "ticks": 8, "read": True,
         "residual": False, "clipped": False},
        # The same scene solved to a residual: hundreds of contact passes in one tick.
        {"name": "cubes_1k_residual", "kind": "cubes", "bodies": 1000, "warm": 30, "ticks": 2, "read": False,
         "residual": True, "clipped": False},
        # The 100,000-body scene (20% hollow cylinders, 400k colliders) in flight: the ticks most of
        # its trajectory consists of.
        {"name": "grid_100k", "kind": "grid", "nx": 50, "ny": 40, "nz": 50, "warm": 6, "ticks": 4},
        # The same scene from its overlapping start: 14M candidate pairs in the first tick.
        {"name": "grid_100k_start", "kind": "grid", "nx": 50, "ny": 40, "nz": 50, "warm": 0, "ticks": 2},
        # 100,000 one-metre cubes at rest on each other: a million touching pairs in every tick.
        {"name": "dense_100k", "kind": "dense", "bodies": 100000, "warm": 20, "ticks": 4},
        # 4,000 five-body bearing chains, a tenth of them closed to loops, in the default closure solve.
        {"name": "chains_4k", "kind": "chains", "chains": 4000, "links": 5, "closed": 0.1, "pcg": False,
         "warm": 4, "ticks": 4},
        # Many independent scenes of 64 to 8,192 bodies stepped by one handle (training environments),
        # closures by PCG to a residual.
        {"name": "batch_64", "kind": "batch", "scenes": 64, "warm": 6, "ticks": 4},
        # One mechanism of 100,000 bodies and 98,010 loop closures.
        {"name": "loops_100k", "kind": "loops", "width": 100, "height": 100, "depth": 10, "warm": 2, "ticks": 2},
        # Key-value sort of millions of 63-bit keys.
        {"name": "sort_5m", "kind": "sort", "n": 5_000_003, "bits": 63},
        # Box pairs as a broadphase hands them over.
        {"name": "sat_1m", "kind": "sat", "n": 1_000_003},
        # Warm-start predictions for a heavy tick's contacts (one output column).
        {"name": "mlp_forward_300k", "kind": "mlp_forward", "n": 300_001, "cols": 1},
        # Training of the warm-start network at the batch its trainer uses.
        {"name": "mlp_train", "kind": "mlp_train", "n": 65_536, "batch": 8192, "steps": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cubes", "grid", "dense", "chains", "batch", "loops", "sort", "sat", "mlp_forward",
                       "mlp_train"])
    if kind == "cubes":
        residual = rng.random() < 0.3
        return {"kind": kind, "bodies": _log_int(rng, 64, 1000 if residual else 4096), "warm": rng.randrange(1, 60),
                "ticks": rng.randrange(1, 3) if residual else rng.randrange(1, 9), "read": rng.random() < 0.5,
                "residual": residual, "clipped": not residual and rng.random() < 0.3}
    if kind == "grid":
        start = rng.random() < 0.3
        return {"kind": kind, "nx": rng.randrange(8, 51), "ny": rng.randrange(4, 41), "nz": rng.randrange(8, 51),
                "warm": 0 if start else rng.randrange(3, 20), "ticks": rng.randrange(1, 3 if start else 5)}
    if kind == "dense":
        return {"kind": kind, "bodies": _log_int(rng, 1024, 100_000), "warm": rng.randrange(1, 40),
                "ticks": rng.randrange(1, 5)}
    if kind == "chains":
        return {"kind": kind, "chains": _log_int(rng, 40, 4000), "links": rng.randrange(3, 7),
                "closed": round(rng.uniform(0.0, 0.15), 3), "pcg": rng.random() < 0.5,
                "warm": rng.randrange(1, 20), "ticks": rng.randrange(1, 4)}
    if kind == "batch":
        return {"kind": kind, "scenes": rng.randrange(2, 65), "warm": rng.randrange(3, 12),
                "ticks": rng.randrange(1, 5)}
    if kind == "loops":
        return {"kind": kind, "width": rng.randrange(5, 101), "height": rng.randrange(5, 101),
                "depth": rng.randrange(1, 11), "warm": rng.randrange(0, 4), "ticks": rng.randrange(1, 3)}
    if kind == "sort":
        return {"kind": kind, "n": _log_int(rng, 500, 5_000_000), "bits": rng.choice([24, 30, 39, 48, 63])}
    if kind == "sat":
        return {"kind": kind, "n": _log_int(rng, 500, 1_000_000)}
    if kind == "mlp_forward":
        return {"kind": kind, "n": _log_int(rng, 100, 300_000), "cols": rng.choice([1, 3, 16])}
    n = _log_int(rng, 1000, 65_536)
    return {"kind": kind, "n": n, "batch": min(n, _log_int(rng, 500, 8192)), "steps": rng.randrange(1, 17)}


# ------------------------------------------------------------------ scenes
def _pow2(n):
    return 1 << max(12, int(n - 1).bit_length())


def _scene(case, seed):
    """(scene or list of scenes, config, pair capacity)"""
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    cfg = GpuPhysicsConfig()
    if kind == "cubes":
        n = case["bodies"]
        scene = scenes.falling_cubes(n, seed=seed, box=10.0 * (n / 1000.0) ** (1.0 / 3.0))
        cfg = learned.residual_config() if case["residual"] else GpuPhysicsConfig(
            contact_manifold=abi.MANIFOLD_CLIPPED if case["clipped"] else abi.MANIFOLD_POINT)
        pairs = _pow2(64 * n)
    elif kind == "grid":
        scene = scenes.stack_grid(case["nx"], case["ny"], case["nz"], seed=seed)
        pairs = _pow2(160 * scene.body_count)
    elif kind == "dense":
        scene = scenes.dense_grid(case["bodies"])
        scene.velocities["linear"][:, :3] = rng.normal(0.0, 0.02, (scene.body_count, 3))
        pairs = _pow2(20 * scene.body_count)
    elif kind == "chains":
        scene = scenes.bearing_chains(case["chains"], case["links"], seed=seed, closure_fraction=case["closed"])
        if case["pcg"]:
            cfg = learned.closure_config()
        pairs = _pow2(32 * scene.body_count)
    elif kind == "batch":
        # the sizes of scenes.batched_uneven, the same for every seed; the scenes are the seed's
        scene = [scenes.mixed_scene(int(64 * 128 ** u), seed + i)
                 for i, u in enumerate(scenes.Rng(0).uniform("batch_sizes", case["scenes"]))]
        cfg = learned.closure_config()
        pairs = _pow2(160 * sum(s.body_count for s in scene))
    else:
        # the seed places the lattice; quarter metres keep its coordinates exact in 32 bits
        place = rng.integers(1, 100, 2) * 0.25
        scene = scenes.translated(scenes.loops_grid(case["width"], case["height"], case["depth"]),
                                  (place[0], 0.0, place[1]))
        pairs = _pow2(32 * scene.body_count)
    return scene, cfg, pairs


class _Rows:
    """Device rows of a handle as a CUDA array; keeps the handle alive."""

    def __init__(self, gpu, address, rows, cols):
        self._gpu = gpu
        self.__cuda_array_interface__ = {"shape": (rows, cols), "typestr": "<f4", "data": (int(address), False),
                                         "version": 2}


class Simulation:
    """A handle with the state that its passes start from."""

    def __init__(self, case, seed):
        scene, cfg, pairs = _scene(case, seed)
        caps = {"pair_capacity": pairs}
        if isinstance(scene, list):
            gpu = GpuPhysics.batch(scene, cfg, capacities=caps)
            q = sum(s.coordinate_count for s in scene)
        else:
            gpu = GpuPhysics(scene, cfg, capacities=caps)
            q = scene.coordinate_count
        for tick in range(1, case["warm"] + 1):
            gpu.dispatch_tick(tick)
        gpu.wait()
        self.gpu, self.ticks, self.read = gpu, case["ticks"], case.get("read", False)
        st, n = gpu.state_buffers(), gpu.body_count()
        rows = [(st.positions, n, 4), (st.rotations, n, 4), (st.linear_velocities, n, 4),
                (st.angular_velocities, n, 4)] + ([(st.coordinates, q, 2)] if q else [])
        self.live = [torch.as_tensor(_Rows(gpu, a, r, c), device="cuda") for a, r, c in rows]
        self.saved = [t.clone() for t in self.live]
        self.stream = torch.cuda.ExternalStream(int(st.stream))
        self.hosts = [np.zeros(n, abi.TRANSFORM) for _ in range(self.ticks)] if self.read else []
        torch.cuda.synchronize()


def _run_ticks(sim):
    with torch.cuda.stream(sim.stream):
        torch._foreach_copy_(sim.live, sim.saved)
    for tick in range(1, sim.ticks + 1):
        sub = sim.gpu.dispatch_tick(tick)
        if sim.read:
            sim.gpu.read_snapshot_transforms(sub.snapshot_slot, sim.hosts[tick - 1])
    last = sim.gpu.read_last_tick()
    return {"counts": [last.error_flags, last.pair_count, last.contact_count, last.active_contact_count,
                       last.closure_iterations, last.contact_iterations],
            "state": sim.live, "snapshots": [h.view(np.float32) for h in sim.hosts]}


# -------------------------------------------------------------- operations
def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _sort_inputs(case, seed):
    n, g = case["n"], _generator(seed)
    keys = torch.randint(0, min(1 << case["bits"], (1 << 63) - 1), (n,), dtype=torch.int64, device="cuda", generator=g)
    return keys, torch.arange(n, dtype=torch.int32, device="cuda")


def _sat_inputs(case, seed):
    """Boxes of about a quarter metre whose centres lie about one box apart."""
    n, g = case["n"], _generator(seed)

    def boxes(center):
        q = torch.randn((n, 4), device="cuda", generator=g)
        x, y, z, w = (q / q.norm(dim=1, keepdim=True)).unbind(1)
        out = torch.zeros((n, 4, 4), device="cuda")
        out[:, 0, :3] = center
        out[:, 1, :3] = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y + w * z), 2 * (x * z - w * y)], 1)
        out[:, 2, :3] = torch.stack([2 * (x * y - w * z), 1 - 2 * (x * x + z * z), 2 * (y * z + w * x)], 1)
        out[:, 3, :3] = torch.stack([2 * (x * z + w * y), 2 * (y * z - w * x), 1 - 2 * (x * x + y * y)], 1)
        out[:, :3, 3] = 0.05 + 0.15 * torch.rand((n, 3), device="cuda", generator=g)
        return out

    center = 4.0 * torch.randn((n, 3), device="cuda", generator=g)
    return boxes(center), boxes(center + 0.16 * torch.randn((n, 3), device="cuda", generator=g))


def _mlp_inputs(case, seed):
    n, g = case["n"], _generator(seed)
    params = torch.from_numpy(init_params(seed % (1 << 31), out_scale=1.0)).cuda()
    x = torch.randn((n, 16), device="cuda", generator=g)
    t = torch.zeros((n, 16), device="cuda")
    t[:, 0] = torch.sin(x[:, 0]) + 0.5 * x[:, 1] * x[:, 2]
    w = torch.zeros(16, device="cuda")
    w[0] = 1.0
    return params, x, t, w


LEARNING_RATE = 2e-3


def prepare(case, seed):
    kind = case["kind"]
    if kind in TICK_KINDS:
        return Simulation(case, seed)
    state = {"case": case}
    if kind == "sort":
        state["keys"], state["values"] = _sort_inputs(case, seed)
    elif kind == "sat":
        state["a"], state["b"] = _sat_inputs(case, seed)
    else:
        state["params"], state["x"], state["t"], state["w"] = _mlp_inputs(case, seed)
        state["m"], state["v"] = torch.zeros_like(state["params"]), torch.zeros_like(state["params"])
        state["ws"] = ops.MlpWorkspace(case.get("batch", case["n"]))
    return state


def run(state):
    if isinstance(state, Simulation):
        return _run_ticks(state)
    case, s = state["case"], state
    if case["kind"] == "sort":
        return ops.sort_keys(s["keys"], s["values"], key_bits=case["bits"])
    if case["kind"] == "sat":
        return ops.obb_sat(s["a"], s["b"])
    if case["kind"] == "mlp_forward":
        return ops.mlp_forward(s["params"], s["x"], y_cols=case["cols"], ws=s["ws"])
    losses = ops.mlp_train(s["params"], s["m"], s["v"], s["x"], s["t"], s["w"], steps=case["steps"],
                           batch=case["batch"], lr=LEARNING_RATE, ws=s["ws"])
    return {"params": s["params"], "m": s["m"], "v": s["v"], "losses": losses}


# ------------------------------------------------------------- 64-bit values
def _exact_sat(a, b):
    """First axis (A0 B0 A1 B1 A2 B2, then Ai x Bj) with a negative penetration, else the
    smallest penetration; the normal points from A to B."""
    a, b = a.double(), b.double()
    ax, bx = a[:, 1:4, :3], b[:, 1:4, :3]
    ah, bh = a[:, :3, 3], b[:, :3, 3]
    delta = b[:, 0, :3] - a[:, 0, :3]
    raws = []
    for i in range(3):
        raws += [ax[:, i], bx[:, i]]
    for i in range(3):
        for j in range(3):
            raws.append(torch.linalg.cross(ax[:, i], bx[:, j]))
    n = len(delta)
    best = torch.full((n,), float("inf"), dtype=torch.float64, device=a.device)
    normal = torch.zeros((n, 3), dtype=torch.float64, device=a.device)
    normal[:, 0] = 1.0
    done = torch.zeros(n, dtype=torch.bool, device=a.device)
    for raw in raws:
        l2 = (raw * raw).sum(1)
        axis = raw / l2.clamp_min(1e-30).sqrt()[:, None]
        sd = (delta * axis).sum(1)
        pen = ((ax * axis[:, None]).sum(2).abs() * ah).sum(1) + ((bx * axis[:, None]).sum(2).abs() * bh).sum(1) \
            - sd.abs()
        axis = torch.where((sd < 0)[:, None], -axis, axis)
        valid = l2 >= 1e-10
        early = ~done & valid & (pen < 0)
        take = ~done & valid & (early | (pen < best))
        best = torch.where(take, pen, best)
        normal = torch.where(take[:, None], axis, normal)
        done = done | early
    return torch.cat([normal, best[:, None]], 1)


def _unpack(p):
    return p[:1024].view(64, 16), p[1024:5120].view(64, 64), p[5120:6144].view(16, 64), p[6144:6208], p[6208:6224]


def _exact_forward(p, x):
    w1, w2, w3, b2, b3 = _unpack(p)
    x = x.clone()
    x[:, 15] = 1.0
    h = torch.relu(torch.relu(x @ w1.T) @ w2.T + b2)
    return h @ w3.T + b3


def _exact_train(case, p, x, t, w):
    p, x, t, w = (v.double() for v in (p, x, t, w))
    m, v, losses, at = torch.zeros_like(p), torch.zeros_like(p), [], 0
    n, batch = case["n"], case["batch"]
    for k in range(1, case["steps"] + 1):
        if at + batch > n:
            at = 0
        q = p.clone().requires_grad_(True)
        y = _exact_forward(q, x[at:at + batch])
        loss = ((y - t[at:at + batch]) ** 2 * w).sum() / batch
        (g,) = torch.autograd.grad(loss, q)
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        p = p - LEARNING_RATE * (m / (1 - 0.9 ** k)) / ((v / (1 - 0.999 ** k)).sqrt() + 1e-8)
        losses.append(loss.detach())
        at += batch
    return {"params": p, "m": m, "v": v, "losses": torch.stack(losses)}


def exact(case, seed):
    kind = case["kind"]
    if kind in TICK_KINDS:
        # a tick's contact set is decided by comparisons and its relaxed-Jacobi passes amplify
        # rounding, so 64 bits give another trajectory, not this one's limit
        return None
    if kind == "sort":
        keys, values = _sort_inputs(case, seed)
        k, order = torch.sort(keys, stable=True)
        return k, values[order]
    if kind == "sat":
        return _exact_sat(*_sat_inputs(case, seed)), None
    p, x, t, w = _mlp_inputs(case, seed)
    if kind == "mlp_forward":
        return _exact_forward(p.double(), x.double())[:, :case["cols"]]
    return _exact_train(case, p, x, t, w)


# -------------------------------------------------------------------- work
def _counts(case):
    """(bodies, colliders, bearings) of a tick case, as its generator makes them on average."""
    kind = case["kind"]
    if kind in ("cubes", "dense"):
        return case["bodies"], case["bodies"], 0
    if kind == "grid":
        n = case["nx"] * case["ny"] * case["nz"]
        return n, 4 * n, 0
    if kind == "chains":
        n = case["chains"] * case["links"]
        return n, n, case["chains"] * (case["links"] - 1 + case["closed"])
    if kind == "batch":
        n = 1675 * case["scenes"]
        return n, 4 * n, n // 60
    w, h, d = case["width"], case["height"], case["depth"]
    return w * h * d, w * h * d, (2 * w * h - w - h) * d + d - 1


def work(case):
    """Bytes: body state, masses and snapshot, collider and bearing rows once per tick; an
    operation's inputs and outputs.  Flops: a tick's contacts are not known here."""
    kind = case["kind"]
    if kind in TICK_KINDS:
        b, c, j = _counts(case)
        return {"bytes": case["ticks"] * (b * (64 + 64 + 64 + 8 + 32) + c * 64 + j * 80), "flops": 0}
    n = case["n"]
    if kind == "sort":
        return {"bytes": 24 * n, "flops": 0}
    if kind == "sat":
        return {"bytes": (128 + 20) * n, "flops": 15 * 60 * n}
    per_sample = 2 * (16 * 64 + 64 * 64 + 64 * 16)
    if kind == "mlp_forward":
        return {"bytes": (64 + 4 * case["cols"]) * n, "flops": per_sample * n}
    samples = case["steps"] * case["batch"]
    return {"bytes": 128 * samples + 24 * 6224, "flops": 3 * per_sample * samples}
