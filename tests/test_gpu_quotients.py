"""The grouped quotients of the block assembly, the factorisation and the body finish, at operands
inside their range, at its edges and outside it (where the plain division runs): bodies from very
light to very heavy, whose masses over dt^2 are the divisors and numerators. Every state is the
oracle's, bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("density", [1e-16, 1e-13, 1e-10, 1.0, 1e7, 1e9, 1e13, 1e20])
def test_mass_range(pkg, gpu, oracle, density):
    capi = pkg.capi
    rng = np.random.default_rng(5)
    n = 7
    size = np.concatenate([[[30, 30, 1]], rng.uniform(0.5, 1.5, (n, 3))])
    position = np.concatenate([[[0, 0, -0.5]], np.stack([np.zeros(n), np.zeros(n), 0.9 + 1.6 * np.arange(n)], 1)])
    velocity = np.concatenate([[[0, 0, 0]], rng.uniform(-1, 1, (n, 3))])
    d = [0.0] + [density * 3.0**k for k in range(n)]
    states = []
    for api in (gpu, oracle):
        w = capi.World(api)
        w.add_bodies(capi.make_body_descs(size, d, 0.5, position, velocity=velocity))
        run = []
        for _ in range(40):
            w.step()
            run.append(w.state())
        states.append(run)
    for a, b in zip(*states):
        for x, y in zip(a, b):
            assert np.array_equal(x, y, equal_nan=True)


def test_equal_to_division(pkg, tmp_path):
    """`quotient` itself beside the compiler's division, compiled with the library's flags: 16 million pairs over its
    range, with all-ones and short mantissas and at the range's ends, zeros of both signs; and that it refuses what
    is outside its range and nothing inside it."""
    import ctypes
    import os
    import subprocess

    from avbd_gb300 import build

    here = os.path.dirname(os.path.abspath(__file__))
    lib = str(tmp_path / "quotients.so")
    subprocess.run([build.nvcc()] + build.NVCC_FLAGS + ["-I" + build.CSRC, "-shared", os.path.join(here, "cuda", "quotients.cu"), "-o", lib],
                   check=True)
    out = (ctypes.c_ulonglong * 4)()
    assert ctypes.CDLL(lib).check_quotients(out) == 0
    wrong, refused, taken_outside, taken = out
    assert (wrong, refused, taken_outside) == (0, 0, 0) and taken > 10_000_000
