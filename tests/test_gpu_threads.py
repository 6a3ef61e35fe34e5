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


@pytest.mark.parametrize("code", [BINS], ids=["bins"])
def test_threads(code):
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=900, cwd=ROOT)
    assert r.returncode == 0, r.stderr[-800:]
