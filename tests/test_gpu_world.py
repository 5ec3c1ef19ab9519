"""The step's second half as one launch, a cluster per world: worlds around its limits (bodies a
CTA, contact tasks, worlds whose parts do not fit in shared memory, many worlds in one store) against
the oracle, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(api, capi, descs, steps, params=None, interleaved=None, room=0):
    p = api.default_params()
    for k, v in (params or {}).items():
        setattr(p, k, v)
    w = capi.World(api, p, max_bodies=max(len(descs), room))
    w.add_bodies(descs)
    out = []
    for _ in range(steps):
        if interleaved:
            w.step_interleaved(*interleaved)
        else:
            w.step()
        out.append(w.state())
    return out


def same(a, b):
    return all(np.array_equal(x, y, equal_nan=True) for s, t in zip(a, b) for x, y in zip(s, t))


def heap(capi, n, seed, spread=1.0):
    """`n` boxes of unequal size and random orientation in a loose heap on a ground."""
    rng = np.random.default_rng(seed)
    size = rng.uniform(0.4, 1.2, (n, 3))
    q = rng.normal(size=(n, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    side = max(1, int(np.ceil((n / 3.0) ** 0.5)))
    i = np.arange(n)
    pos = np.stack([spread * (i % side), spread * (i // side % side), 0.8 + 1.1 * (i // (side * side))], 1)
    pos += rng.uniform(-0.05, 0.05, pos.shape)
    return capi.make_body_descs(np.concatenate([[[80, 80, 1]], size]), [0.0] + [1.0] * n, 0.5,
                                np.concatenate([[[0, 0, -0.5]], pos]), np.concatenate([[[0, 0, 0, 1]], q]),
                                np.concatenate([[[0, 0, 0]], rng.uniform(-1, 1, (n, 3))]))


# One CTA, two, the odd sizes around a CTA's share of the bodies, the largest cluster.
@pytest.mark.parametrize("n", [1, 2, 23, 24, 25, 49, 97, 193, 385, 700])
def test_sizes(pkg, gpu, oracle, n):
    capi = pkg.capi
    d = heap(capi, n, n)
    assert same(run(gpu, capi, d, 25), run(oracle, capi, d, 25))


# Bodies inside one another: far more manifolds a body than the shared-memory form holds, in the first
# step (before any count is known) and after.
@pytest.mark.parametrize("n,spread", [(150, 0.25), (260, 0.12)])
def test_dense_world_does_not_fit(pkg, gpu, oracle, n, spread):
    capi = pkg.capi
    d = heap(capi, n, 3, spread)
    room = 16384  # the store is sized by this: eight manifolds and sixteen pairs a body
    assert same(run(gpu, capi, d, 6, room=room), run(oracle, capi, d, 6))


@pytest.mark.parametrize("params,interleaved", [
    ({"jacobian_rebuild_distance": 0.02}, None), ({"jacobian_rebuild_distance": 0.05, "dt": 1 / 120}, (2, 3)),
    ({"position_projection": 0}, None), ({"speculative_margin": 0.0}, None), ({"newton_ratio": 0.5}, None),
    ({"adaptive_beta": 1, "iterations": 3}, (3, 2))])
def test_options(pkg, gpu, oracle, params, interleaved):
    capi = pkg.capi
    d = heap(capi, 120, 9)
    assert same(run(gpu, capi, d, 20, params, interleaved), run(oracle, capi, d, 20, params, interleaved))


def test_many_worlds_added_and_removed(pkg, gpu):
    """A store that starts too large to be kept in world order, then loses worlds until it is, then gains
    one: each world equals the same world alone."""
    capi = pkg.capi
    worlds, n = 500, 140
    b = capi.Batch(gpu.lib, max_worlds=worlds, max_bodies=worlds * (n + 1))
    kinds = [heap(capi, n, s) for s in range(5)]
    add = lambda d: (b._api.check(b.fn["batch_add_world"](b.handle, len(d), d, 0, None, capi.C.byref(capi.C.c_int()))),
                     b.sizes.append(len(d)))
    for w in range(worlds):
        add(kinds[w % 5])
    b.step(8)
    b.remove_worlds([w for w in range(worlds) if w % 10])
    b.step(8)
    add(kinds[0])
    b.step(8)
    alone = [run(gpu, capi, d, 24) for d in kinds]
    for w in range(0, 50, 7):
        assert same([b.state(w)], [alone[w * 10 % 5][23]])
    assert same([b.state(50)], [alone[0][7]])


# One wide dynamic plate (first or last in the store) under many small boxes: more adjacency entries than
# a thread sorts, more partners of one body than the pair stash holds, and none.
@pytest.mark.parametrize("boxes,last", [(20, False), (90, False), (90, True), (200, True)])
def test_wide_plate(pkg, gpu, oracle, boxes, last):
    capi = pkg.capi
    rng = np.random.default_rng(boxes)
    side = int(np.ceil(boxes ** 0.5))
    i = np.arange(boxes)
    pos = np.stack([0.6 * (i % side), 0.6 * (i // side), 1.0 + 0 * i], 1) + rng.uniform(-0.02, 0.02, (boxes, 3))
    size, density = [[0.4, 0.4, 0.4]] * boxes, [1.0] * boxes
    plate = [[0.6 * side + 2, 0.6 * side + 2, 0.3]], [5.0], [[0.3 * side, 0.3 * side, 0.45]]
    ground = [[60, 60, 1]], [0.0], [[0, 0, -0.5]]
    parts = [ground, (size, density, pos.tolist()), plate] if last else [ground, plate, (size, density, pos.tolist())]
    d = capi.make_body_descs(*[sum((list(p[k]) for p in parts), []) for k in (0, 1)], 0.5,
                             sum((list(p[2]) for p in parts), []))
    assert same(run(gpu, capi, d, 25), run(oracle, capi, d, 25))


def tangle(capi, n, seed, ragdolls=True):
    """A heap with every kind of force among its bodies: a hub that carries most of them (more terms
    than a warp has lanes), chains, world anchors, springs and, with `ragdolls`, soft joints and
    free, limited and sprung rotations (of which the oracle may have other last bits)."""
    d = heap(capi, n, seed)
    at = lambda i: np.array(d[i].position[:])
    lock, free = (1, 0, 0, 0, 0, 0), (0, 0, 0, 0, 0, 0)
    hinge = free if ragdolls else lock
    rng = np.random.default_rng(seed)
    forces = []
    for i in range(2, n + 1):
        a = 1 if i % 2 else i - 1  # the hub, or a chain
        r = tuple(0.5 * (at(i) - at(a)))
        ends = (a, i, r, tuple(-x for x in r))
        kind = i % 7
        if kind == 0:
            forces.append(("spring", *ends, 40.0, -1.0 if i % 3 else 0.7))
        elif kind == 1:
            forces.append(("generic", *ends, (lock, lock, lock, hinge, lock, lock)))
        elif kind == 2 and ragdolls:
            forces.append(("generic", *ends, (lock, lock, (0, 0, 0, 60.0, 0.1, 1.5), (2, -0.3, 0.3, 0, 0, 0),
                                              (0, 0, 0, 40.0, 0.2, 2.0), lock)))
        elif kind == 3:
            forces.append(("generic", -1, i, tuple(at(i)), (0.0, 0.0, 0.0), (lock, (2, -0.5, 0.1, 0, 0, 0), free, hinge, hinge, hinge)))
        elif kind == 4:
            forces.append((*ends, *((800.0, 30.0) if ragdolls else (float("inf"), 0.0)), float("inf")))
        elif kind == 5 and rng.random() < 0.5:
            forces.append(("ignore", a, i))
        else:
            forces.append((*ends, float("inf"), 0.0, float("inf")))
    return d, forces


def run_forces(api, capi, world, params, steps=20, interleaved=None):
    d, forces = world
    p = api.default_params()
    for k, v in params.items():
        setattr(p, k, v)
    w = capi.World(api, p, max_bodies=16384, max_forces=max(1, len(forces)))
    w.add_bodies(d)
    for f in forces:
        w.add_force(f)
    out = []
    for _ in range(steps):
        w.step_interleaved(*interleaved) if interleaved else w.step()
        out.append(w.state())
    return out


# Forces on one CTA and on two, against the oracle.
@pytest.mark.parametrize("n", [2, 9, 47])
def test_forces(pkg, gpu, oracle, n):
    capi = pkg.capi
    world = tangle(capi, n, n, ragdolls=False)
    assert same(run_forces(gpu, capi, world, {}), run_forces(oracle, capi, world, {}))


# Every force, up to the largest cluster, arms kept from the dual, substeps, no projection: the same bits
# as the separate launches.
@pytest.mark.parametrize("n,params,interleaved", [
    (12, {}, None), (47, {}, None), (200, {}, None), (400, {}, None), (130, {"jacobian_rebuild_distance": 0.05}, None),
    (60, {"iterations": 3, "position_projection": 0}, (2, 3))])
def test_forces_as_separate_launches(pkg, gpu, monkeypatch, n, params, interleaved):
    capi = pkg.capi
    world = tangle(capi, n, n)
    here = run_forces(gpu, capi, world, params, interleaved=interleaved)
    monkeypatch.setenv("AVBDG_NO_WORLD", "1")
    assert same(here, run_forces(gpu, capi, world, params, interleaved=interleaved))


# The colouring by a block a world: more bodies than its threads, every body coloured or those with forces,
# the same bits as across the store.
@pytest.mark.parametrize("params", [{}, {"contact_only_overflow": 0}])
@pytest.mark.parametrize("n", [1025, 2600])
def test_colouring(pkg, gpu, monkeypatch, n, params):
    capi = pkg.capi
    d, forces = tangle(capi, n, n)
    world = d, forces[:60] + forces[-40:]
    here = run_forces(gpu, capi, world, params, steps=8)
    monkeypatch.setenv("AVBDG_NO_WORLD", "1")
    assert same(here, run_forces(gpu, capi, world, params, steps=8))


# Some worlds of very different sizes, up to 128 bodies a CTA, without forces and with: each equals itself alone.
@pytest.mark.parametrize("forces", [False, True])
@pytest.mark.parametrize("worlds,most", [(4, 1700), (16, 900), (30, 480)])
def test_some_worlds(pkg, gpu, worlds, most, forces):
    capi = pkg.capi
    kinds = [tangle(capi, max(2, int(most * k / worlds) - k % 3), k) for k in range(worlds, 0, -1)]
    kinds = [(d, f[:25] if forces and k % 3 else []) for k, (d, f) in enumerate(kinds)]
    b = capi.Batch(gpu.lib, max_worlds=worlds, max_bodies=4 * sum(len(d) for d, _ in kinds), max_forces=25 * worlds)
    for d, f in kinds:
        b._api.check(b.fn["batch_add_world"](b.handle, len(d), d, len(f), capi.make_force_descs(f), capi.C.byref(capi.C.c_int())))
        b.sizes.append(len(d))
    b.step(10)
    for w in range(0, worlds, 3 if worlds > 4 else 1):
        assert same([b.state(w)], run_forces(gpu, capi, kinds[w], {}, steps=10)[9:])


# The phase times of a step (one launch a world, or the separate launches): all parts counted, and together
# no more than the host waited.
@pytest.mark.parametrize("separate", ["0", "1"])
def test_phase_times(pkg, gpu, monkeypatch, separate):
    import time

    monkeypatch.setenv("AVBDG_NO_WORLD", separate)
    capi = pkg.capi
    w = capi.World(gpu, gpu.default_params(), max_bodies=301)
    w.add_bodies(heap(capi, 300, 5))
    for _ in range(12):
        begin = time.perf_counter()
        w.step()
        wall = 1000 * (time.perf_counter() - begin)
        st = w.stats()
        parts = [st.broad_ms, st.graph_ms, st.solve_ms] + ([st.finish_ms] if separate == "1" else [])
        assert min(parts) > 0 and abs(sum(parts) - st.total_ms) < 1e-9 and 0.05 < st.total_ms < wall


def press(capi, layers, anchors):
    """Plates held by ball joints to the world (`anchors` of them each), `layers` of 34 boxes between them. The plates
    come last, so all take the first colour."""
    rng = np.random.default_rng(7)
    i = np.arange(34)
    size, pos = [], []
    for k in range(layers):
        pos.append(np.stack([0.9 * (i % 7) - 2.7, 0.9 * (i // 7) - 1.8, 0.5 + 0.99 * k + 0 * i], 1) + [0.01, 0.01, 0] * rng.uniform(-1, 1, (34, 3)))
        size += [[0.6, 0.6, 0.6]] * 34
    plates = [[0, 0, 0.99 * k] for k in range(layers + 1)]
    size += [[8, 6, 0.4]] * (layers + 1)
    d = capi.make_body_descs(size, [1.0] * len(size), 0.5, np.concatenate(pos + [plates]))
    forces = []
    for k, n in enumerate(anchors):
        for _ in range(n):
            r = rng.uniform([-4, -3, -0.2], [4, 3, 0.2])
            forces.append((-1, 34 * layers + k, tuple(r + plates[k]), tuple(r), 2000.0, 0.0, float("inf")))
    return d, forces


# A CTA (65 to 72 bodies: 288 terms a pass) whose first colour takes three passes and more, with a body that comes
# over from the pass before beside one that goes on to the next, both cut inside a manifold's contacts.
def test_colour_of_many_passes(pkg, gpu, oracle):
    capi = pkg.capi
    d, forces = press(capi, 2, (17, 10, 10))
    worlds = 78  # more than half the SMs: a CTA a world
    b = capi.Batch(gpu.lib, max_worlds=worlds, max_bodies=worlds * len(d), max_forces=worlds * len(forces))
    for _ in range(worlds):
        b._api.check(b.fn["batch_add_world"](b.handle, len(d), d, len(forces), capi.make_force_descs(forces), capi.C.byref(capi.C.c_int())))
        b.sizes.append(len(d))
    w = capi.World(oracle, oracle.default_params())
    w.add_bodies(d)
    for f in forces:
        w.add_force(f)
    cut = 0
    for _ in range(24):
        b.step()
        w.step()
        for k in (0, 40, 77):
            assert same([b.state(k)], [w.state()])
        m, (colour, ids) = w.manifolds(), w.colours()
        assert (colour[ids >= 68] == 0).all()
        terms = [3 * n + m["count"][(m["body_a"] == 68 + k) | (m["body_b"] == 68 + k)].sum() for k, n in enumerate((17, 10, 10))]
        ends = np.cumsum(terms)
        cut += ends[0] < 288 < ends[1] < 576 < ends[2]
    assert cut > 12  # steps that cross both borders


# Substeps without the brake, whose barriers otherwise part a substep's rebase from the next one's warm start: one
# CTA and several, without forces and with.
@pytest.mark.parametrize("interleaved", [(2, 3), (4, 2)])
@pytest.mark.parametrize("n", [20, 45, 300])
def test_substeps_without_brake(pkg, gpu, oracle, n, interleaved):
    capi, params = pkg.capi, {"speculative_margin": 0.0}
    d = heap(capi, n, n)
    assert same(run(gpu, capi, d, 20, params, interleaved), run(oracle, capi, d, 20, params, interleaved))
    world = tangle(capi, n, n, ragdolls=False)
    world = world[0], world[1][:30]
    assert same(run_forces(gpu, capi, world, params, interleaved=interleaved), run_forces(oracle, capi, world, params, interleaved=interleaved))


# A world that does not fit in shared memory, with substeps (each begins from the gaps that the rebase of the one before
# wrote in the same launch): arms kept or not, sleepers, and with forces, where jointed bodies find no colour free and the
# oracle has other last bits: the same as the separate launches.
@pytest.mark.parametrize("forces", [False, True])
@pytest.mark.parametrize("params", [{}, {"jacobian_rebuild_distance": 0.05},
                                    {"sleep_frames": 2, "sleep_linear_threshold": 5.0, "sleep_angular_threshold": 5.0}])
def test_dense_world_with_substeps(pkg, gpu, oracle, monkeypatch, params, forces):
    capi = pkg.capi
    dense = heap(capi, 150, 3, 0.25)
    for i in range(1, 151):
        dense[i].sleep_mode = i % 3 if "sleep_frames" in params else 0
    world = dense, tangle(capi, 150, 3, ragdolls=False)[1][:12] if forces else []
    here = run_forces(gpu, capi, world, params, steps=6, interleaved=(3, 2))
    monkeypatch.setenv("AVBDG_NO_WORLD", "1")
    assert same(here, run_forces(gpu, capi, world, params, steps=6, interleaved=(3, 2)))
    if not forces:
        assert same(here, run_forces(oracle, capi, world, params, steps=6, interleaved=(3, 2)))


# A step's phases by either route: the brake counts with the warm start ("graph"), a chain of 300 candidates here, and the
# adjacency that a new force makes a step rebuild first counts with the broad phase.
@pytest.mark.parametrize("separate", ["0", "1"])
def test_brake_and_adjacency_phases(pkg, gpu, monkeypatch, separate):
    from test_gpu_waits import approaching_column

    monkeypatch.setenv("AVBDG_NO_WORLD", separate)
    capi = pkg.capi

    def least(margin):
        p = gpu.default_params()
        p.speculative_margin = margin
        w = capi.World(gpu, p, max_bodies=301)
        w.add_bodies(approaching_column(pkg, 300))
        begin = w.state()
        begin[2][:] = [0, 0, 0]
        times = []
        for _ in range(12):
            w.set_state(*begin)
            w.step()
            times.append(w.stats().graph_ms)
        return min(times)

    assert least(0.05) - least(0.0) > 0.05
    w = pkg.scenes.instantiate(gpu, pkg.scenes.lattice(nx=40, ny=40, nz=16))
    w.step(3)
    fresh, plain = [], []
    for k in range(8):
        w.add_ignore_collision(1 + 2 * k, 2 + 2 * k)
        w.step()
        fresh.append(w.stats().broad_ms)
        w.step()
        plain.append(w.stats().broad_ms)
    assert np.median(fresh) - np.median(plain) > 0.008  # its seven launches take 2 us each at least


# Profiled steps of a world that is otherwise stepped in one launch: each kernel timed, the state the same.
def test_profiled_world(pkg, gpu, monkeypatch):
    monkeypatch.setenv("AVBDG_NO_TUNE", "1")
    capi = pkg.capi
    worlds = [capi.World(gpu, gpu.default_params(), max_bodies=301) for _ in range(2)]
    for w in worlds:
        w.add_bodies(heap(capi, 300, 5))
        w.step(4)
    worlds[0].set_profiling(True)
    for w in worlds:
        w.step(6)
    kt, rounds = worlds[0].take_kernel_times(), gpu.default_params().iterations
    assert (kt.steps, kt.manifold_launches, kt.body_launches, kt.narrow_launches) == (6, 6 * rounds, 6 * rounds, 6)
    assert min(kt.manifold_ms, kt.body_ms, kt.narrow_ms) > 0
    worlds[0].set_profiling(False)
    for w in worlds:
        w.step(4)
    assert same([worlds[0].state()], [worlds[1].state()]) and worlds[0].stats().kernel_launches == worlds[1].stats().kernel_launches


# A step timed by two events around its launches: no less than its kernels' own clock shows, no more than the host waited.
@pytest.mark.parametrize("graphs", ["0", "1"])
def test_step_events(pkg, gpu, monkeypatch, graphs):
    import time

    monkeypatch.setenv("AVBDG_STEP_EVENTS", "1")
    monkeypatch.setenv("AVBDG_NO_GRAPHS", graphs)
    capi = pkg.capi
    w = capi.World(gpu, gpu.default_params(), max_bodies=301)
    w.add_bodies(heap(capi, 300, 5))
    for _ in range(12):
        begin = time.perf_counter()
        w.step()
        wall = 1000 * (time.perf_counter() - begin)
        st = w.stats()
        assert 0.95 * (st.broad_ms + st.graph_ms + st.solve_ms + st.finish_ms) < st.total_ms < wall
