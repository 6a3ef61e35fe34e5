"""GPU: wf_stats.launches counts the kernels of a ray query."""
import numpy as np
import pytest

from wavefrontpathtracing_gb300 import Renderer, scenes
from tests.helpers import load_scene_into
from tests.test_gpu_trace import random_rays

pytestmark = pytest.mark.gpu


def test_reordered_trace_counts_its_kernels():
    rays = random_rays(5000, 0.0, 1.0, seed=3)
    with Renderer(8, 8) as r:
        load_scene_into(r, scenes.box_scene(8, 8, subdivision=1))
        hits = r.trace(rays)
        assert r.stats()["launches"] == 1
        again = r.trace(rays, reorder=True)
        # keys, decision, two sort passes of five kernels, the traversal
        assert r.stats()["launches"] == 2 + 2 * 5 + 1
        assert np.array_equal(hits.view(np.uint8), again.view(np.uint8))
