"""The work that programs have this library do, as cases that can be timed and compared.

A case is a dict of plain values. `listed()` names the standing ones, `draw(rng)` gives another of
the same ranges, `prepare` makes what a program has in hand before the call, `run` is one pass
through the public entry points (the C ABI through its ctypes binding), `work` counts what a pass
cannot do without, and `exact` gives the outputs in 64 bits where a closed form exists.

Kinds of case:
  world  one world. A pass restores saved poses and velocities, steps, and reads the bodies back:
         a tick of a game server that writes its bodies and reads their transforms (1 tick), or a
         rollback, replay or planning rollout from a saved state (several).
  batch  many independent worlds in one store, stepped together from a saved state: training
         environments, parameter sweeps.
  serve  requests of mixed size that arrive while others run, stepped by continuous batching.
  query  many ray picks and one box query against a world.
  sort   the standalone sort + unique of 64-bit keys in device memory.
"""

import ctypes
import importlib
import math
from types import SimpleNamespace

import numpy as np
import torch

pkg = importlib.import_module("godot-avbd_gb300")
capi = importlib.import_module("godot-avbd_gb300.capi")

BODY = np.dtype([("size", "f4", 3), ("shape", "i4"), ("density", "f4"), ("friction", "f4"), ("position", "f4", 3),
                 ("orientation", "f4", 4), ("velocity", "f4", 3), ("angular_velocity", "f4", 3), ("layer", "u4"),
                 ("mask", "u4"), ("lock_linear", "u4"), ("lock_angular", "u4"), ("sleep_mode", "u4")])
assert BODY.itemsize == ctypes.sizeof(capi.BodyDesc)
INF = float("inf")


# ------------------------------------------------------------------------------------------------
# Cases
# ------------------------------------------------------------------------------------------------

def listed():
    return [
        # The smallest call there is: a stack of boxes in one world, one server tick. Launches and
        # latency are all of it.
        {"name": "tick_stack16", "kind": "world", "scene": "stack", "n": 16, "ticks": 1},
        # The benchmark's 420-box pyramid (two 20-row walls), an eight-tick rollback.
        {"name": "walls420", "kind": "world", "scene": "walls", "rows": 20, "walls": 2, "ticks": 8},
        # The benchmark's mass-ratio pile with its hard ball-jointed chain: coloured Gauss-Seidel and
        # block Jacobi in one world.
        {"name": "pile1653_chain32", "kind": "world", "scene": "pile", "n": 1653, "chain": 32, "ticks": 4},
        # The reference's own diagnostic settings: a wall dropped on a wall at 240 Hz in four
        # interleaved substeps of two rounds, with the arm cache.
        {"name": "drop420_substeps", "kind": "world", "scene": "drop", "rows": 20, "ticks": 2, "substeps": 4,
         "rounds": 2},
        # A game level: sleeping walls, spheres, cylinders, ragdolls of ball and generic joints,
        # springs, ignore pairs, a few bodies that never sleep.
        {"name": "level600", "kind": "world", "scene": "level", "n": 600, "ticks": 2},
        # A world of odd size between the small ones and the lattice.
        {"name": "lattice_13x17x11", "kind": "world", "scene": "lattice", "nx": 13, "ny": 17, "nz": 11, "ticks": 4},
        # The largest single world of the benchmark: 65,536 boxes.
        {"name": "lattice_64x64x16", "kind": "world", "scene": "lattice", "nx": 64, "ny": 64, "nz": 16, "ticks": 2},
        # Training environments of ordinary size.
        {"name": "envs256", "kind": "batch", "worlds": 256, "n_min": 8, "n_max": 64, "ticks": 4},
        # The benchmark's batch: 4096 worlds of 8 to 512 boxes, walls and mass-ratio piles.
        {"name": "envs4096", "kind": "batch", "worlds": 4096, "n_min": 8, "n_max": 512, "ticks": 2},
        # A burst of requests, two arriving at each tick, with and without joints.
        {"name": "serve32", "kind": "serve", "requests": 32, "n_min": 16, "n_max": 2048, "steps_min": 8,
         "steps_max": 40},
        # Mouse picks, line-of-sight and sensor rays of one frame against a pile-sized world.
        {"name": "query4096", "kind": "query", "n": 1653, "rays": 4096},
        # The broad phase's pair sort on a caller's own keys.
        {"name": "sort_1m", "kind": "sort", "count": 1 << 20, "bits": 43, "repeat": 2, "static": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stack", "walls", "pile", "drop", "level", "lattice", "batch", "batch", "serve", "query", "sort"])
    ticks = rng.randint(1, 8)
    if kind == "stack":
        return {"kind": "world", "scene": "stack", "n": _log_int(rng, 2, 64), "ticks": ticks}
    if kind == "walls":
        return {"kind": "world", "scene": "walls", "rows": rng.randint(3, 20), "walls": rng.randint(1, 4), "ticks": ticks}
    if kind == "pile":
        return {"kind": "world", "scene": "pile", "n": _log_int(rng, 16, 4000), "chain": rng.choice([0, 0, 4, 9, 32]),
                "ticks": ticks}
    if kind == "drop":
        return {"kind": "world", "scene": "drop", "rows": rng.randint(4, 20), "ticks": rng.randint(1, 3),
                "substeps": rng.choice([2, 3, 4]), "rounds": rng.randint(2, 4)}
    if kind == "level":
        return {"kind": "world", "scene": "level", "n": _log_int(rng, 60, 3000), "ticks": rng.randint(1, 4)}
    if kind == "lattice":
        nz = rng.randint(3, 16)
        side = [_log_int(rng, 3, 64) for _ in range(2)]
        return {"kind": "world", "scene": "lattice", "nx": side[0], "ny": side[1], "nz": nz, "ticks": rng.randint(1, 2)}
    if kind == "batch":
        lo = _log_int(rng, 4, 16)
        return {"kind": "batch", "worlds": _log_int(rng, 16, 4000), "n_min": lo, "n_max": _log_int(rng, 2 * lo, 512),
                "ticks": rng.randint(1, 2)}
    if kind == "serve":
        lo = rng.randint(1, 12)
        return {"kind": "serve", "requests": _log_int(rng, 4, 40), "n_min": 16, "n_max": _log_int(rng, 100, 2048),
                "steps_min": lo, "steps_max": lo + rng.randint(1, 28)}
    if kind == "query":
        return {"kind": "query", "n": _log_int(rng, 20, 4000), "rays": _log_int(rng, 1, 8192)}
    static = rng.random() < 0.3
    return {"kind": "sort", "count": _log_int(rng, 1000, 1 << 18 if static else 1 << 21), "bits": rng.randint(24, 64),
            "repeat": rng.randint(1, 8), "static": static}


# ------------------------------------------------------------------------------------------------
# Scenes (packed body records, creation order; the seed moves positions and velocities)
# ------------------------------------------------------------------------------------------------

def _boxes(n, size=(1, 1, 1), density=1.0, friction=0.5):
    b = np.zeros(n, BODY)
    b["size"], b["density"], b["friction"] = size, density, friction
    b["orientation"][:, 3] = 1.0
    b["layer"] = b["mask"] = 1
    return b


def _ground(extent, friction=0.5, thickness=1.0):
    g = _boxes(1, (extent, extent, thickness), 0.0, friction)
    g["position"][0, 2] = -0.5 * thickness
    return g


def _shake(rng, b, position=0.005, velocity=0.05):
    b["position"] += rng.uniform(-position, position, b["position"].shape).astype("f4")
    b["velocity"] += rng.uniform(-velocity, velocity, b["velocity"].shape).astype("f4")
    return b


def _wall_cells(rows):
    """Row and place within the row of each box of a wall of `rows` rows, bottom row first."""
    row = np.repeat(np.arange(rows), rows - np.arange(rows))
    return row, np.arange(row.size) - np.repeat(np.cumsum(rows - np.arange(rows)) - (rows - np.arange(rows)),
                                                rows - np.arange(rows))


def _wall(rows, y=0.0, height=1.0, pitch=None, z0=0.0, density=1.0):
    row, k = _wall_cells(rows)
    b = _boxes(row.size, (1, 1, height), density)
    b["position"][:, 0] = (k - (rows - 1 - row) * 0.5) * 1.01
    b["position"][:, 1] = y
    b["position"][:, 2] = z0 + 0.5 * height + row * (height if pitch is None else pitch)
    return b


def _quats(rng, n):
    q = rng.normal(size=(n, 4))
    return (q / np.linalg.norm(q, axis=1, keepdims=True)).astype("f4")


def _pile(rng, n):
    """Boxes with log-uniform edges (0.25 to 2 m) and densities (100 to 1e4), each in its own cell of
    a grid, random orientations."""
    b = _boxes(n)
    b["size"] = np.exp(rng.uniform(math.log(0.25), math.log(2.0), (n, 3)))
    b["density"] = np.exp(rng.uniform(math.log(100.0), math.log(1e4), n))
    b["orientation"] = _quats(rng, n)
    cell = 3.5
    side = max(2, math.ceil((n / 2.0) ** (1.0 / 3.0)))
    i = np.arange(n)
    at = np.stack([i % side, i // side % side, i // (side * side)], axis=1)
    slack = 0.5 * cell - 0.5 * np.linalg.norm(b["size"], axis=1, keepdims=True)
    b["position"] = (at + 0.5) * cell + rng.uniform(-1, 1, (n, 3)) * slack
    b["position"][:, :2] -= 0.5 * side * cell
    return b, side * cell


def _ball(a, b, ra, rb):
    return (a, b, ra, rb, INF, 0.0, INF)


def _chain(first, x, links):
    """A static anchor (body `first`) with `links` links on hard ball joints."""
    b = _boxes(links + 1, (0.2, 0.2, 1.0), 1000.0)
    b["density"][0] = 0.0
    b["position"][:, 0] = x
    b["position"][:, 2] = links + 4.0 - np.arange(links + 1)
    return b, [_ball(first + i, first + i + 1, (0, 0, -0.5), (0, 0, 0.5)) for i in range(links)]


PLAIN = {"gravity": -9.81, "iterations": 10, "dt": float(np.float32(1.0) / np.float32(60.0))}


def _scene(case, rng):
    """(body records, forces, solver fields, ticks to settle) of a one-world case."""
    s = case["scene"]
    if s == "stack":
        b = _boxes(case["n"])
        b["position"][:, 2] = np.arange(case["n"]) * 1.02 + 0.52
        return np.concatenate([_ground(100), _shake(rng, b)]), [], PLAIN, 40
    if s == "walls":
        y = (np.arange(case["walls"]) - 0.5 * (case["walls"] - 1)) * 3.0
        return np.concatenate([_ground(100)] + [_shake(rng, _wall(case["rows"], v)) for v in y]), [], PLAIN, 40
    if s == "pile":
        b, width = _pile(rng, case["n"])
        parts, forces = [_ground(400), b], []
        if case["chain"]:
            links, forces = _chain(1 + case["n"], width, case["chain"])
            parts.append(_shake(rng, links, 0.0))
        return np.concatenate(parts), forces, PLAIN, 150
    if s == "drop":
        low, high = (_wall(case["rows"], 0.0, 0.5, 0.52, z, 2.0) for z in (0.0, 0.52 * case["rows"] + 1.0))
        b = np.concatenate([_ground(80), _shake(rng, low), _shake(rng, high)])
        return b, [], {"gravity": -9.8, "dt": float(np.float32(1.0) / np.float32(240.0)), "iterations": 12, "beta_lin": 1e5,
                       "speculative_margin": 0.02, "jacobian_rebuild_distance": 0.02, "position_projection": 1,
                       "projection_max_correction": 0.1, "contact_only_overflow": 1, "sleep_frames": 30}, 40
    if s == "lattice":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        at = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 3)
        b = _boxes(len(at), friction=0.6)
        b["position"] = (at - [(nx - 1) * 0.5, (ny - 1) * 0.5, 0]) * 1.05 + [0, 0, 0.55] + rng.uniform(-0.02, 0.02, at.shape)
        return np.concatenate([_ground(500, 0.6), b]), [], PLAIN, 60
    return _level(case["n"], rng)


def _level(n, rng):
    parts, forces, count = [_ground(400)], [], 1
    free, lock = (0, 0, 0, 0, 0, 0), (1, 0, 0, 0, 0, 0)
    rows = max(3, min(12, int(math.sqrt(n / 6))))
    per = rows * (rows + 1) // 2
    walls = max(1, int(0.6 * n / per))
    for w in range(walls):  # walls that have come to rest and sleep
        b = _shake(rng, _wall(rows, 3.0 * w), 0.002, 0.0)
        b["sleep_mode"] = 1
        parts.append(b)
        count += len(b)
    dolls = max(1, int(0.15 * n / 6))
    for i in range(dolls):  # ragdolls: a trunk, a head on a ball joint, four limbs on limited hinges
        at = np.array([30.0 + 3.0 * (i % 10), 3.0 * (i // 10), 2.5])
        b = _boxes(6, (0.3, 0.3, 0.8), 100.0)
        b["size"][0], b["size"][1] = (0.6, 0.3, 0.9), (0.3, 0.3, 0.3)
        off = np.array([(0, 0, 0), (0, 0, 0.7), (0.6, 0, 0.1), (-0.6, 0, 0.1), (0.25, 0, -0.95), (-0.25, 0, -0.95)])
        b["position"] = at + off
        parts.append(_shake(rng, b, 0.0, 0.3))
        forces.append(_ball(count, count + 1, (0, 0, 0.5), (0, 0, -0.2)))
        for k in range(2, 6):
            forces.append(("generic", count, count + k, tuple(off[k] * 0.7), tuple(-off[k] * 0.3),
                           (lock, lock, lock, (2, -0.8, 0.8, 0, 0, 0), lock, lock if k < 4 else free)))
            forces.append(("ignore", count, count + k))
        count += 6
    hangs = max(1, int(0.05 * n / 5))
    for i in range(hangs):  # weights on springs
        b = _boxes(5, (0.4, 0.4, 0.4))
        b["density"][0] = 0.0
        b["position"] = np.array([-20.0 - 2.0 * (i % 10), 2.0 * (i // 10), 9.0]) - np.arange(5)[:, None] * [0, 0, 1.2]
        parts.append(_shake(rng, b, 0.0))
        for k in range(4):
            forces.append(("spring", count + k, count + k + 1, (0, 0, -0.15), (0, 0, 0.2), 300.0, -1.0))
        count += 5
    rest = max(4, n - count)
    b = _boxes(rest, (0.4, 0.4, 0.8))  # spheres (radius), cylinders (radius, height) and boxes, dropped
    b["shape"] = np.arange(rest) % 3
    b["orientation"] = _quats(rng, rest)
    i = np.arange(rest)
    b["position"] = np.stack([-5.0 - 1.5 * (i % 8), 1.5 * (i // 8 % 8), 1.0 + 1.5 * (i // 64)], axis=1)
    b["sleep_mode"] = i % 4 != 0
    parts.append(_shake(rng, b, 0.1, 0.5))
    return np.concatenate(parts), forces, dict(PLAIN, sleep_frames=30), 60


def _descs(bodies):
    return (capi.BodyDesc * len(bodies)).from_buffer(np.ascontiguousarray(bodies))


def _params(api, fields):
    p = api.default_params()
    for k, v in fields.items():
        setattr(p, k, v)
    return p


def _sizes(case, count):
    """Log-uniform body counts, the case's own: the seed moves bodies, not sizes."""
    u = np.random.default_rng([case["n_min"], case["n_max"], count]).random(count)
    return np.exp(math.log(case["n_min"]) + u * math.log(case["n_max"] / case["n_min"])).round().astype(int)


def _worlds(case, rng):
    """Body records of every world of a batch, one after another, and where each begins: log-uniform
    sizes, half walls and half piles, each on its own ground."""
    n = _sizes(case, case["worlds"])
    parts = []
    pile, _ = _pile(rng, int(n.max()))
    walls = {}
    for k, size in enumerate(n):
        if k % 2:
            rows = min(20, max(2, round((math.sqrt(8 * size + 1) - 1) / 2)))
            if rows not in walls:
                walls[rows] = _wall(rows)
            parts += [_GROUND, walls[rows]]
        else:
            side = max(2, math.ceil((size / 2.0) ** (1.0 / 3.0)))
            b = pile[rng.integers(0, len(pile), size)]
            i = np.arange(size)
            b["position"] = (np.stack([i % side, i // side % side, i // (side * side)], axis=1) + 0.5) * 3.5
            parts += [_GROUND, b]
    ends = np.cumsum([len(a) + len(b) for a, b in zip(parts[::2], parts[1::2])])
    bodies = np.concatenate(parts)
    moving = bodies["density"] > 0
    bodies["position"][moving] += rng.uniform(-0.005, 0.005, (int(moving.sum()), 3)).astype("f4")
    bodies["velocity"][moving] += rng.uniform(-0.05, 0.05, (int(moving.sum()), 3)).astype("f4")
    return bodies, np.concatenate([[0], ends])


_GROUND = _ground(200)


# ------------------------------------------------------------------------------------------------
# A pass
# ------------------------------------------------------------------------------------------------

def prepare(case, seed):
    rng = np.random.default_rng([seed & 0x7FFFFFFF, 17])
    s = SimpleNamespace(case=case)
    if case["kind"] == "world":
        bodies, forces, fields, settle = _scene(case, rng)
        s.world = _one_world(bodies, forces, fields)
        _tick(s.world, case, settle)
        s.saved = s.world.state()
        s.out = tuple(np.empty_like(a) for a in s.saved)
        s.sleepers = bool(bodies["sleep_mode"].any())
    elif case["kind"] == "batch":
        bodies, ends = _worlds(case, rng)
        s.lib = pkg.load_library()
        s.batch = capi.Batch(s.lib, _params(pkg.gpu_api(), PLAIN), case["worlds"], len(bodies), 0)
        descs, at = _descs(bodies), ctypes.c_int()
        for lo, hi in zip(ends[:-1].tolist(), ends[1:].tolist()):
            rc = s.batch.fn["batch_add_world"](s.batch.handle, hi - lo, ctypes.cast(ctypes.byref(descs, lo * BODY.itemsize),
                                               ctypes.POINTER(capi.BodyDesc)), 0, None, ctypes.byref(at))
            pkg.gpu_api().check(rc)
            s.batch.sizes.append(hi - lo)
        s.batch.step(100)
        s.saved = s.batch.state_all()
        s.out = tuple(np.empty_like(a) for a in s.saved)
    elif case["kind"] == "serve":
        s.server = capi.Server(pkg.load_library(), _params(pkg.gpu_api(), PLAIN), budget_bytes=16 * 10**9, max_resident=64)
        s.requests = [_request(case, k, int(n), rng) for k, n in enumerate(_sizes(case, case["requests"]))]
    elif case["kind"] == "query":
        bodies, origins, dirs, box = _query(case, rng)
        s.world = _one_world(bodies, [], PLAIN)
        s.origins, s.dirs, s.box = origins, dirs, box
    else:
        s.keys = _keys(case, seed)
        s.fn = getattr(pkg.load_library(), "avbdg_sort_unique_keys" + ("_static" if case["static"] else ""))
        s.fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int), ctypes.c_void_p]
    return s


def run(s):
    case = s.case
    if case["kind"] == "world":
        s.world.set_state(*s.saved)
        _tick(s.world, case, case["ticks"])
        out = s.world.state(s.out)
        return (out, s.world.sleeping()) if s.sleepers else out
    if case["kind"] == "batch":
        s.batch.set_state_all(*s.saved)
        s.batch.step(case["ticks"])
        return s.batch.state_all(s.out)
    if case["kind"] == "serve":
        ids, left, got = [], list(s.requests), {}
        while len(got) < len(s.requests):
            for descs, forces, steps in left[:2]:
                ids.append(s.server.admit(SimpleNamespace(n=len(descs), joints=[None] * forces[1]), steps, descs, forces[0]))
            del left[:2]
            if s.server.tick():
                got.update(s.server.results())
        return tuple(np.concatenate([got[i][k] for i in ids]) for k in range(4))
    if case["kind"] == "query":
        body, local = s.world.pick(s.origins, s.dirs)
        found = s.world.collect_aabb(*s.box)
        return body, local, np.concatenate([found, np.full(case["n"] - len(found), -1, found.dtype)])
    keys, count = s.keys.clone(), ctypes.c_int()
    pkg.gpu_api().check(s.fn(keys.data_ptr(), keys.numel(), case["bits"], ctypes.byref(count), None))
    return keys[:count.value]


def _one_world(bodies, forces, fields):
    api = pkg.gpu_api()
    w = capi.World(api, _params(api, fields), max_bodies=len(bodies), max_forces=len(forces))
    w.add_bodies(_descs(bodies))
    for f in forces:
        w.add_force(f)
    return w


def _tick(world, case, ticks):
    if "substeps" in case:
        for _ in range(ticks):
            world.step_interleaved(case["substeps"], case["rounds"])
    else:
        world.step(ticks)


def _request(case, k, n, rng):
    """Request k, about n bodies: walls, or a pile with a short chain, and its step count."""
    forces = []
    if k % 2:
        rows = int(min(20, max(2, math.sqrt(2 * n))))
        walls = max(1, round(n / (rows * (rows + 1) / 2)))
        parts = [_ground(400)] + [_shake(rng, _wall(rows, 1.6 * (w - 0.5 * walls))) for w in range(walls)]
    else:
        b, width = _pile(rng, n)
        links, forces = _chain(1 + n, width, 8)
        parts = [_ground(400), b, links]
    steps = case["steps_min"] + k * 7 % (case["steps_max"] - case["steps_min"] + 1)
    return _descs(np.concatenate(parts)), (capi.make_force_descs(forces), len(forces)), steps


def _query(case, rng):
    """Boxes and spheres on a grid, unit rays between random points around them, one box."""
    b, width = _pile(rng, case["n"])
    b["shape"] = rng.random(len(b)) < 0.25
    b["size"][b["shape"] == 1] *= 0.5
    top = float(b["position"][:, 2].max()) + 2.0
    lo, hi = np.array([-0.6 * width, -0.6 * width, 0.0]), np.array([0.6 * width, 0.6 * width, top])
    o = rng.uniform(lo, hi, (case["rays"], 3)).astype("f4")
    d = rng.uniform(lo, hi, (case["rays"], 3)) - o
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    half = 0.3 * (hi - lo)
    mid = rng.uniform(lo + half, hi - half)
    return b, o, d.astype("f4"), ((mid - half).astype("f4"), (mid + half).astype("f4"))


def _keys(case, seed):
    """Every one of count / repeat distinct keys of `bits` bits, `repeat` times or once more, shuffled."""
    n = max(1, case["count"] // case["repeat"])
    g = torch.Generator(device="cuda").manual_seed(seed)
    keys = torch.arange(n, device="cuda") * -0x61C8864680B583EB + seed  # odd factor: distinct
    if case["bits"] < 64:
        keys &= (1 << case["bits"]) - 1
    return keys[torch.randperm(case["count"], generator=g, device="cuda") % n].contiguous()


# ------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ------------------------------------------------------------------------------------------------

def _size_of(case):
    """Bodies (expected, where they are drawn) of a case."""
    if case["kind"] == "world":
        s = case["scene"]
        if s in ("walls", "drop"):
            return case.get("walls", 2) * case["rows"] * (case["rows"] + 1) // 2 + 1
        return case["nx"] * case["ny"] * case["nz"] + 1 if s == "lattice" else case["n"] + case.get("chain", 0) + 1
    mean = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
    return int((mean + 1) * case.get("worlds", case.get("requests", 1)))


def work(case):
    if case["kind"] == "sort":
        n = case["count"]
        return {"bytes": 16 * n + 16 * n, "flops": n * math.log2(max(n, 2))}
    if case["kind"] == "query":
        n, r = case["n"], case["rays"]
        return {"bytes": 64 * n + 40 * r, "flops": 60.0 * r * math.log2(max(n, 2))}
    n = _size_of(case)
    if case["kind"] == "serve":
        ticks, rounds = 0.5 * (case["steps_min"] + case["steps_max"]), 10
    else:
        ticks = case["ticks"]
        rounds = case["substeps"] * case["rounds"] if "substeps" in case else 10
    # Per body and tick: pose, velocity and step-start velocity in and out (116 B each way) and its
    # constants (48 B); about two manifolds of four contacts a body, each with its pair, key, arms,
    # penalty and force in and out. Per round: about 450 operations a contact (dual and next stamps,
    # both sides) and 700 a body (block assembly and 6x6 solve). Poses and velocities cross to the
    # host and back once a pass.
    contacts = 8 * n
    return {"bytes": ticks * (n * 280 + 2 * contacts * 60) + 2 * 52 * n,
            "flops": ticks * rounds * (450.0 * contacts + 700.0 * n)}


# ------------------------------------------------------------------------------------------------
# The same in 64 bits
# ------------------------------------------------------------------------------------------------

def exact(case, seed):
    # A step takes thousands of branches on its contacts and carries every rounding on: it has no
    # closed form, and a 64-bit restatement of the solver would be a second solver.
    if case["kind"] == "sort":
        flip = torch.tensor(-(1 << 63), device="cuda")
        return torch.unique(_keys(case, seed) ^ flip) ^ flip
    if case["kind"] != "query":
        return None
    bodies, origins, dirs, _ = _query(case, np.random.default_rng([seed & 0x7FFFFFFF, 17]))
    dev = {"device": "cuda", "dtype": torch.float64}
    q = torch.tensor(bodies["orientation"], **dev)
    x = torch.tensor(bodies["position"], **dev)
    size = torch.tensor(bodies["size"], **dev)
    ball = torch.tensor(bodies["shape"] == 1, device="cuda")

    def turn(v):  # into every body's frame: (rays, 3) or (rays, bodies, 3)
        u = -q[:, :3].expand(*v.shape[:-1], 3)
        t = 2 * torch.linalg.cross(u, v)
        return v + q[:, 3:] * t + torch.linalg.cross(u, t)

    ids, local = [], []
    for k in range(0, len(origins), 512):
        o = torch.tensor(origins[k:k + 512], **dev)[:, None, :] - x
        o, d = turn(o), turn(torch.tensor(dirs[k:k + 512], **dev)[:, None, :].expand(*o.shape))
        a, b = (-0.5 * size - o) / d, (0.5 * size - o) / d
        near, far = torch.minimum(a, b).amax(-1).clamp(min=0.0), torch.maximum(a, b).amin(-1)
        t = torch.where((near <= far) & (far >= 0), near, INF)
        half = (o * d).sum(-1)
        disc = half * half - (o * o).sum(-1) + size[:, 0] ** 2
        root = disc.clamp(min=0).sqrt()
        s = torch.where(-half - root >= 0, -half - root, -half + root)
        t = torch.where(ball, torch.where((disc >= 0) & (s >= 0), s, INF), t)
        best = t.argmin(1)
        row = torch.arange(len(best), device="cuda")
        hit = torch.isfinite(t[row, best])
        ids.append(torch.where(hit, best, -1).to(torch.int32))
        local.append(torch.where(hit[:, None], o[row, best] + d[row, best] * t[row, best].where(hit, torch.zeros((), **dev))[:, None], 0.0))
    return torch.cat(ids), torch.cat(local), None
