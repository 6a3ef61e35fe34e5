"""GPU: TLAS builds whose working set comes close to the 48 KiB of shared memory
that a block has without asking for more: a kernel's own variables lie beside
it.  In a process of its own, sizes ascending, so that no larger build has asked
before; then from two threads with sizes on either side."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CODE = """
import sys, threading
import numpy as np
import wavefrontpathtracing_gb300 as wf
from oracle import oracle as orc
from tests.test_gpu_tlas_walk import lattice_instances
metric = int(sys.argv[1])
failed = []

def build(r, n, compare=False):
    inst = lattice_instances(n, seed=n)
    try:
        blob = r.tlas_build(inst)
        if compare and not np.array_equal(blob, orc.tlas_build(inst, metric=metric)):
            failed.append((n, "differs"))
    except wf.WFError as e:
        failed.append((n, str(e)))

with wf.Renderer(8, 8, tlas_metric=metric) as r:
    for n in [*range(440, 660, 3), *range(1480, 1560)]:
        build(r, n, n % 16 == 0)

def work(n):
    with wf.Renderer(8, 8, tlas_metric=metric) as r:
        for _ in range(60):
            build(r, n)

threads = [threading.Thread(target=work, args=(n,)) for n in (1100, 1250, 1900, 2040)]
for t in threads: t.start()
for t in threads: t.join()
assert not failed, failed[:5]
"""


@pytest.mark.parametrize("metric", [0, 1, 2, 3])
def test_builds_near_the_default_shared_memory(metric):
    r = subprocess.run([sys.executable, "-c", CODE, str(metric)], capture_output=True, text=True, timeout=600, cwd=ROOT)
    assert r.returncode == 0, r.stderr[-800:]
