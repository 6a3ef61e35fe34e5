"""GPU: the adjoint's recorded hits.  Where the memory limit leaves no room for
a whole wave's hits the waves get shorter; the gradients are the same sums in
another order (float atomics): with fewer than 2^17 terms per parameter, each
rounded once per addition, the two differ by far less than 2^17 * 2^-24 of the
sum of the terms' magnitudes, and by 1e-5 relative in the 2-norm here."""
import ctypes

import numpy as np
import pytest

import wavefrontpathtracing_gb300 as wf
from wavefrontpathtracing_gb300 import Renderer, scenes
from tests.helpers import load_scene_into

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nee,rr", [(0, 99), (1, 3)])
def test_short_tape_gives_the_same_gradients(nee, rr):
    desc = scenes.box_scene(64, 64, subdivision=1)
    rng = np.random.default_rng(3)
    dloss = rng.normal(size=(64, 64, 3)).astype(np.float32)
    kw = dict(max_bounces=6, spp=20, frame_seed=9, nee=nee, rr_start_depth=rr)
    L = wf.load()
    grads = []
    for limited in (False, True):
        with Renderer(64, 64) as r:   # capacity 65,536 paths: a whole tape 9.2 MB, the shortest 2 MB
            load_scene_into(r, desc)
            r.set_albedo(np.random.default_rng(5).uniform(0.1, 0.9, size=(r.scene_triangle_count(), 3)))
            r.render(max_bounces=1, spp=1)
            r.synchronize()
            used = ctypes.c_uint64()
            try:
                if limited:
                    wf.check(L.wf_get_device_memory_usage(ctypes.byref(used)))
                    wf.check(L.wf_set_device_memory_limit(used.value + (5 << 20)))
                first = r.adjoint(dloss, **kw)
                again = r.adjoint(dloss, **kw)
            finally:
                L.wf_set_device_memory_limit(0)
            for a, b in zip(first, again):
                assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(a)
            grads.append(first)
            launches = r.stats()["launches"]
        if limited:
            assert launches > whole_launches   # more, shorter waves
        else:
            whole_launches = launches
    for a, b in zip(*grads):
        assert np.isfinite(a).all() and np.linalg.norm(a) > 0.0
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(a)
