"""Scratch that calls keep: the sort's block of a device and the query blocks of a world, over sizes that
grow, shrink and pass what is kept, on several threads and streams."""

import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def sorter(pkg):
    fn = pkg.load_library().avbdg_sort_unique_keys
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.POINTER(ctypes.c_int), ctypes.c_void_p]
    fn.restype = ctypes.c_int
    return fn


def sorted_unique(fn, keys, stream=None):
    import torch

    with torch.cuda.stream(stream):
        t = torch.from_numpy(keys.view(np.int64)).cuda()
    out = ctypes.c_int(-1)
    assert fn(t.data_ptr(), keys.size, 64, ctypes.byref(out), stream.cuda_stream if stream else None) == 0
    if stream:
        stream.synchronize()
    return t.cpu().numpy().view(np.uint64)[: out.value]


# 9 million keys take more than is kept.
def test_sort_sizes(pkg):
    fn, rng = sorter(pkg), np.random.default_rng(1)
    for n in (1000, 500_000, 3, 9_000_000, 70_000):
        keys = rng.integers(0, 1 << 40, n, dtype=np.uint64)
        assert np.array_equal(sorted_unique(fn, keys), np.unique(keys))


def test_sort_threads_and_streams(pkg):
    import torch

    fn, bad = sorter(pkg), []

    def work(k):
        rng, stream = np.random.default_rng(k), torch.cuda.Stream()
        for n in (200_000, 1000, 900_000, 30_000):
            keys = rng.integers(0, 1 << 30, n + k, dtype=np.uint64)
            if not np.array_equal(sorted_unique(fn, keys, stream), np.unique(keys)):
                bad.append((k, n))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_sort_block_is_given_back(pkg, gpu):
    import torch

    fn = sorter(pkg)
    w = pkg.scenes.instantiate(gpu, pkg.scenes.shape_mix())
    sorted_unique(fn, np.arange(100, dtype=np.uint64))
    w.close()
    before = torch.cuda.mem_get_info()[0]
    w = pkg.scenes.instantiate(gpu, pkg.scenes.shape_mix())
    keys = torch.arange(4_000_000, dtype=torch.int64, device="cuda")
    out = ctypes.c_int()
    assert fn(keys.data_ptr(), keys.numel(), 64, ctypes.byref(out), None) == 0
    w.close()
    del keys
    torch.cuda.empty_cache()
    assert torch.cuda.mem_get_info()[0] >= before


# 150,000 rays answer in more than is kept for them.
def test_query_sizes(pkg, gpu, oracle):
    scenes = pkg.scenes
    a, b = (scenes.instantiate(x, scenes.shape_mix()) for x in (gpu, oracle))
    a.step(20)
    b.step(20)
    rng = np.random.default_rng(4)
    for n in (1, 500, 7, 150_000, 33, 5000):
        origins = rng.uniform([-15, -6, 1], [15, 6, 8], (n, 3)).astype(np.float32)
        dirs = (rng.uniform([-15, -3, -1], [15, 3, 2], (n, 3)) - origins).astype(np.float32)
        dirs[::2] /= np.linalg.norm(dirs[::2], axis=1, keepdims=True)
        (ga, la), (gb, lb) = (x.pick(origins[:, :], dirs) for x in (a, b))
        assert np.array_equal(ga, gb) and np.array_equal(la, lb)
        box = (-2.0 - n % 5, -2, 0), (1.0 + n % 7, 3, 4)
        assert np.array_equal(a.collect_aabb(*box), b.collect_aabb(*box))


# More than a million pairs, around a tile of 64 bodies; rays of unit length and not, from inside bodies and
# from far away, along axes, one with a NaN and one of length zero.
@pytest.mark.parametrize("n", [63, 64, 65, 300])
def test_pick_tiles(pkg, gpu, oracle, n):
    capi = pkg.capi
    rng = np.random.default_rng(n)
    size, pos = rng.uniform(0.3, 2.0, (n, 3)), rng.uniform(-8, 8, (n, 3))
    q = rng.normal(size=(n, 4))
    d = capi.make_body_descs(size, [1.0] * n, 0.5, pos, q / np.linalg.norm(q, axis=1, keepdims=True))
    for i in range(0, n, 3):
        d[i].shape = 1
    rays = (1 << 20) // n + 77
    origins = rng.uniform(-12, 12, (rays, 3)).astype(np.float32)
    dirs = rng.normal(size=(rays, 3)).astype(np.float32)
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    dirs[::7] = np.eye(3, dtype=np.float32)[rng.integers(0, 3, len(dirs[::7]))]
    dirs[1::7] *= rng.uniform(0.1, 3.0, (len(dirs[1::7]), 1)).astype(np.float32)
    origins[2::7] -= 300 * dirs[2::7]
    origins[3::7] = pos[rng.integers(0, n, len(origins[3::7]))]
    dirs[5], dirs[6] = 0, (np.nan, 1, 0)
    worlds = [capi.World(api, api.default_params(), max_bodies=n) for api in (gpu, oracle)]
    for w in worlds:
        w.add_bodies(d)
    (ga, la), (gb, lb) = (w.pick(origins, dirs) for w in worlds)
    part = [worlds[0].pick(origins[i:i + 1000], dirs[i:i + 1000]) for i in range(0, rays, 1000)]  # a thread a pair
    assert np.array_equal(ga, np.concatenate([p[0] for p in part]))
    assert np.array_equal(la, np.concatenate([p[1] for p in part]), equal_nan=True)
    ga[6], la[6] = gb[6], lb[6]  # which of its distances of NaN a ray takes is not the oracle's
    assert np.array_equal(ga, gb) and np.array_equal(la, lb, equal_nan=True) and (ga >= 0).sum() > rays // 20


# The scan behind a collect, by one block, by a cluster of two to sixteen CTAs and by three launches.
@pytest.mark.parametrize("n", [4095, 4096, 4097, 20_000, 140_000, 540_000])
def test_collect_scans(pkg, gpu, n):
    capi, rng = pkg.capi, np.random.default_rng(n)
    pos = rng.uniform(-50, 50, (n, 3))
    w = capi.World(gpu, gpu.default_params(), max_bodies=n)
    w.add_bodies(capi.make_body_descs([[0.1, 0.1, 0.1]] * n, [1.0] * n, 0.5, pos))
    pos, half = pos.astype(np.float32), np.float32(0.05)
    lo, hi = np.float32([-30, -30.5, -20]), np.float32([25, 35, 41])
    inside = ((pos - half <= hi) & (lo <= pos + half)).all(axis=1)
    assert np.array_equal(w.collect_aabb(lo, hi), np.nonzero(inside)[0][::-1])  # list order: the last first


# The cluster's scan while other work fills the device, so that its CTAs start apart: each of a world's
# collects counts the same bodies, on four streams at once.
def test_scans_on_a_busy_device(pkg, gpu):
    capi, bad = pkg.capi, []

    def work(n):
        rng = np.random.default_rng(n)
        pos = rng.uniform(-50, 50, (n, 3))
        w = capi.World(gpu, gpu.default_params(), max_bodies=n)
        w.add_bodies(capi.make_body_descs([[0.1, 0.1, 0.1]] * n, [1.0] * n, 0.5, pos))
        at, half = pos.astype(np.float32), np.float32(0.05)
        for k in range(200):
            lo = np.float32([-40 + k % 7, -30.5, -20])
            hi = lo + np.float32([50, 60, 40 + k % 11])
            inside = ((at - half <= hi) & (lo <= at + half)).all(axis=1)
            if not np.array_equal(w.collect_aabb(lo, hi), np.nonzero(inside)[0][::-1]):
                bad.append((n, k))
        w.step(20)

    threads = [threading.Thread(target=work, args=(n,)) for n in (4200, 9000, 33_000, 100_000)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
