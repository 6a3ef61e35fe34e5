"""GPU: contexts in threads of their own do not disturb one another.  Each case
runs in a process of its own, so that no earlier call has set anything up."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

COMMON = """
import threading
import numpy as np
import wavefrontpathtracing_gb300 as wf
from wavefrontpathtracing_gb300 import Batch, Renderer, scenes
failed = []

def run(jobs):
    def guard(f, *a):
        try:
            f(*a)
        except Exception as e:
            failed.append((a, repr(e)))
    threads = [threading.Thread(target=guard, args=j) for j in jobs]
    for t in threads: t.start()
    for t in threads: t.join()
    assert not failed, failed[:4]
"""

# builds whose kernels take 8 to 29 KB of shared memory, by the number of bins
BINS = COMMON + """
tris = scenes.triangle_soup(2, seed=1, mu=-2.0)

def work(bins):
    for _ in range(1500):
        with Renderer(16, 16) as r:
            for _ in range(3):
                r.create_mesh_from_triangles(tris, interval_count=bins)

run([(work, b) for b in (64, 2, 53, 4, 60, 3, 48, 2)])
"""

# contexts made while other threads' batches record their graphs
CREATE = COMMON + """
tris = scenes.icosphere(4)

def render(k):
    with Renderer(8, 8) as r:
        mesh = r.create_mesh_from_triangles(tris)
        b = Batch(r)
        b.begin_scene(16, 16, 2, scenes.make_view((0, 0, -4), (0, 0, 0), 60.0, 16, 16), (1.0, 1.0, 1.0))
        b.submit(mesh, np.eye(4))
        b.end_scene()
        first = None
        for i in range(150):
            b.set_config(capacity=1024 + 8 * (i % 2) + k, block=128)   # another graph each time
            b.render(max_bounces=2, frame_seed=3)
            image = b.read_image(0)
            first = image if first is None else first
            assert np.array_equal(image, first)
        b.close()

def make(k):
    for _ in range(300):
        with Renderer(8, 8) as r:
            r.create_mesh_from_triangles(tris)

run([(render, 0), (make, 1), (render, 2), (make, 3), (make, 4)])
"""


@pytest.mark.parametrize("code", [BINS, CREATE], ids=["bins", "create"])
def test_threads(code):
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=900, cwd=ROOT)
    assert r.returncode == 0, r.stderr[-800:]
