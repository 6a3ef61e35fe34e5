"""GPU: the scratch blocks kept between builds: builds of different sizes in
turn, from two threads with a context each, give the blobs that fresh scratch
gives; idle blocks do not count as used memory, make room for an allocation at
the memory limit and go with the last context."""
import ctypes
import threading

import numpy as np
import pytest

import wavefrontpathtracing_gb300 as wf
from wavefrontpathtracing_gb300 import Renderer, scenes

pytestmark = pytest.mark.gpu


def used():
    n = ctypes.c_uint64()
    wf.check(wf.load().wf_get_device_memory_usage(ctypes.byref(n)))
    return n.value


def test_kept_scratch_is_idle_bounded_and_thread_safe(orc):
    sizes = (40, 3000, 20000, 700, 9000)
    soups = [scenes.triangle_soup(n, seed=n, mu=-3.0) for n in sizes]
    want = [orc.bvh_build(t, 16, False, 4) for t in soups]
    errors = []

    def work(order):
        try:
            with Renderer(8, 8) as r:
                for k in order:
                    if not np.array_equal(r.bvh_build(soups[k], 16, False, 4), want[k]):
                        errors.append(k)
        except Exception as e:   # noqa: BLE001 - reported below
            errors.append(e)

    with Renderer(8, 8) as r:
        before = used()
        for k in (2, 0, 4, 2):
            assert np.array_equal(r.bvh_build(soups[k], 16, False, 4), want[k])
            assert used() == before
        threads = [threading.Thread(target=work, args=(o * 3,)) for o in ([0, 1, 2, 3, 4], [4, 2, 3, 0, 1])]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not errors, errors
        # a limit that leaves room for the smallest build's scratch only
        L = wf.load()
        try:
            wf.check(L.wf_set_device_memory_limit(used() + (1 << 20)))
            assert np.array_equal(r.bvh_build(soups[0], 16, False, 4), want[0])
            with pytest.raises(wf.WFError) as e:
                r.bvh_build(soups[2], 16, False, 4)
            assert e.value.status == -2
        finally:
            L.wf_set_device_memory_limit(0)
        assert np.array_equal(r.bvh_build(soups[2], 16, False, 4), want[2])
