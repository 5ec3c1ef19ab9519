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
