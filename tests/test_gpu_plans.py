"""A step's captured graph serves the sizes near it, and a store keeps no more than so many of them."""

import numpy as np
import pytest

from test_gpu_world import heap, same

pytestmark = pytest.mark.gpu


# A world that gains a body every third tick: a plan per class of sizes, not per size; its states are the oracle's.
def test_growing_world(pkg, gpu, oracle, monkeypatch):
    monkeypatch.setenv("AVBDG_NO_TUNE", "1")
    capi = pkg.capi
    first, more = heap(capi, 40, 1), 120
    rng = np.random.default_rng(3)
    extra = capi.make_body_descs(rng.uniform(0.4, 1.0, (more, 3)), [1.0] * more, 0.5,
                                 np.stack([rng.uniform(-2, 6, more), rng.uniform(-2, 6, more), rng.uniform(6, 9, more)], 1))
    worlds = [capi.World(api, api.default_params(), max_bodies=400) for api in (gpu, oracle)]
    eager = 0
    for w in worlds:
        w.add_bodies(first)
    for k in range(more):
        for w in worlds:
            w.add_bodies((capi.BodyDesc * 1)(extra[k]))
            for _ in range(3):
                w.step()
                eager += w is worlds[0] and not w.stats().graph_step
        assert same([worlds[0].state()], [worlds[1].state()])
    # Sizes 42 to 161: thirteen classes, two plans each (a tick after a new body, another tick), by either route.
    assert eager <= 52


# A hundred and fifty plans taken twice each: the first of them is forgotten, and runs again.
def test_plans_are_bounded(pkg, gpu, oracle, monkeypatch):
    monkeypatch.setenv("AVBDG_NO_TUNE", "1")
    capi = pkg.capi
    worlds = [capi.World(api, api.default_params(), max_bodies=64) for api in (gpu, oracle)]
    for w in worlds:
        w.add_bodies(heap(capi, 12, 1))
    for k in range(150):
        for w in worlds:
            for _ in range(2):
                w.step_interleaved(2 + k % 5, 1 + k // 5)
    graphed = worlds[0].stats().graph_step
    for w in worlds:
        w.step_interleaved(2, 1)
    assert graphed and not worlds[0].stats().graph_step
    assert same([worlds[0].state()], [worlds[1].state()])
