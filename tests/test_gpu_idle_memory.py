"""GPU: the blocks that the library keeps between calls are idle: an adjoint's
recorded hits do not count as used, make room for other contexts at the memory
limit and go with their context; at the limit a small build does not take a
large build's block; all go with the last context."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

import wavefrontpathtracing_gb300 as wf
from wavefrontpathtracing_gb300 import Renderer, scenes
from tests.helpers import load_scene_into

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def used():
    n = ctypes.c_uint64()
    wf.check(wf.load().wf_get_device_memory_usage(ctypes.byref(n)))
    return n.value


def limit(n):
    wf.check(wf.load().wf_set_device_memory_limit(n))


def test_adjoint_hits_are_idle_after_the_call():
    torch = pytest.importorskip("torch")
    side, bounces = 256, 6
    capacity = side * side * 16
    tape = capacity * (bounces + 1) * 20   # 147 MB
    desc = scenes.box_scene(side, side, subdivision=1)
    dloss = np.random.default_rng(3).normal(size=(side, side, 3)).astype(np.float32)
    kw = dict(max_bounces=bounces, spp=16, frame_seed=9)

    def frame(r):
        load_scene_into(r, desc)
        r.render(**kw)
        r.synchronize()

    a = Renderer(side, side)
    frame(a)
    a.set_albedo(np.full((a.scene_triangle_count(), 3), 0.5))
    before = used()
    with Renderer(side, side) as b:
        frame(b)
        second = used() - before
    want = a.adjoint(dloss, **kw)
    after = used()
    # the call's other buffers: 16 bytes per path, image gradient, replicas
    assert after - before < 16 * capacity + 16 * side * side + (16 << 20)
    try:
        limit(after + tape // 2 + second)   # no room for the idle hits and a second context
        with Renderer(side, side) as b:
            frame(b)
            got = a.adjoint(dloss, **kw)    # half the hits fit beside it: shorter waves
            assert used() == after + second
    finally:
        limit(0)
    for x, y in zip(want, got):
        assert np.linalg.norm(x - y) <= 1e-5 * np.linalg.norm(x)
    a.adjoint(dloss, **kw)
    with Renderer(8, 8):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        a.close()
        assert torch.cuda.mem_get_info()[0] - free > tape   # with their context, while another lives


def test_small_build_leaves_a_large_block_alone_at_the_limit():
    opts = dict(interval_count=16, max_leaf_prims=4)
    large, small = scenes.triangle_soup(60_000, seed=1, mu=-3.0), scenes.triangle_soup(2_000, seed=2, mu=-3.0)
    with Renderer(8, 8) as r:
        r.bvh_build(small, **opts)
        base = used()
        try:
            # the least room that the large build takes, to 16 KiB
            lo, hi = 0, 64 << 20
            while hi - lo > 1 << 14:
                mid = (lo + hi) // 2
                limit(1)
                limit(base + mid)
                try:
                    r.bvh_build(large, **opts)
                    hi = mid
                except wf.WFError as e:
                    assert e.status == -2
                    lo = mid
            limit(base + hi)
            r.bvh_build(large, **opts)   # its scratch stays, idle, and fills the limit
            r.create_mesh_from_triangles(small, **opts)
        finally:
            limit(0)


LAST = """
import torch
from wavefrontpathtracing_gb300 import Renderer, scenes
with Renderer(8, 8) as r:
    r.bvh_build(scenes.triangle_soup(200_000, seed=1, mu=-3.0), interval_count=16, max_leaf_prims=4)   # 50 MB of scratch
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
assert torch.cuda.mem_get_info()[0] - free > 30 << 20
"""


def test_idle_blocks_go_with_the_last_context():
    pytest.importorskip("torch")
    subprocess.run([sys.executable, "-c", LAST], check=True, timeout=300, cwd=ROOT)
