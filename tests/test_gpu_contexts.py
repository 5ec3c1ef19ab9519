"""Two CUDA contexts on one device, in turn: what a launch may use (shared memory beyond 48 KB, clusters
beyond eight CTAs) is set for each, and scratch kept in one is not lost to the other."""

import contextlib
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

from test_gpu_scratch import sorter
from test_gpu_world import heap, run, run_forces, same, tangle

pytestmark = pytest.mark.gpu


class Contexts:
    def __init__(self):
        self.cu = ctypes.CDLL("libcuda.so.1")
        self.ok(self.cu.cuInit(0))
        self.second = ctypes.c_void_p()
        self.ok(self.cu.cuCtxCreate_v2(ctypes.byref(self.second), 0, 0))
        self.ok(self.cu.cuCtxPopCurrent_v2(ctypes.byref(ctypes.c_void_p())))

    def ok(self, rc):
        assert rc == 0, rc

    @contextlib.contextmanager
    def other(self):
        self.ok(self.cu.cuCtxPushCurrent_v2(self.second))
        try:
            yield
        finally:
            self.ok(self.cu.cuCtxPopCurrent_v2(ctypes.byref(ctypes.c_void_p())))

    def free_bytes(self):
        free, total = ctypes.c_size_t(), ctypes.c_size_t()
        self.ok(self.cu.cuMemGetInfo_v2(ctypes.byref(free), ctypes.byref(total)))
        return free.value

    def upload(self, a):
        p = ctypes.c_uint64()
        self.ok(self.cu.cuMemAlloc_v2(ctypes.byref(p), ctypes.c_size_t(a.nbytes)))
        self.ok(self.cu.cuMemcpyHtoD_v2(p, a.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(a.nbytes)))
        return p

    def download(self, p, a):
        self.ok(self.cu.cuMemcpyDtoH_v2(a.ctypes.data_as(ctypes.c_void_p), p, ctypes.c_size_t(a.nbytes)))
        self.ok(self.cu.cuMemFree_v2(p))


@pytest.fixture(scope="module")
def contexts(gpu):
    import torch

    torch.cuda.init()
    torch.zeros(1, device="cuda")
    c = Contexts()
    yield c
    c.ok(c.cu.cuCtxDestroy_v2(c.second))


# A world in one cluster, a wide colouring, and stores whose scans take a cluster.
def test_worlds_in_two_contexts(pkg, gpu, contexts):
    capi = pkg.capi
    small, (many, forces) = heap(capi, 300, 2), tangle(capi, 2600, 3)

    def steps():
        return run(gpu, capi, small, 8) + run_forces(gpu, capi, (many, forces[:50]), {}, steps=4) + run(gpu, capi, small, 4, room=9000)

    first = steps()
    with contexts.other():
        second = steps()
    assert same(first, second) and same(first, steps())


RESET = """
import ctypes, sys
import __graft_entry__ as entry
pkg = entry.load_package()
gpu, scenes = pkg.gpu_api(), pkg.scenes
def steps():
    w = scenes.instantiate(gpu, scenes.pyramid420())
    w.step(5)
    d = w.digest()
    w.close()
    return d
first = steps()
assert ctypes.CDLL("libcuda.so.1").cuDevicePrimaryCtxReset_v2(0) == 0
assert steps() == first
"""


# After its device was reset a program makes its worlds anew.
def test_world_after_a_device_reset():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", RESET], cwd=root, check=True, timeout=120)


# Sorts in two contexts in turn: each context's block stays its own and is found again.
def test_sort_in_two_contexts(pkg, gpu, contexts):
    fn, rng = sorter(pkg), np.random.default_rng(2)
    free = []
    for turn in range(5):
        for where in (contextlib.nullcontext, contexts.other):
            with where():
                keys = rng.integers(0, 1 << 40, 1_000_000, dtype=np.uint64)
                p, count = contexts.upload(keys), ctypes.c_int()
                assert fn(p.value, keys.size, 40, ctypes.byref(count), None) == 0
                out = np.empty_like(keys)
                contexts.download(p, out)
                assert np.array_equal(out[: count.value], np.unique(keys))
        free.append(contexts.free_bytes())
    assert free[1] == free[4]
