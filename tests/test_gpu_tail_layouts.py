"""GPU: the tail over every BLAS layout.  The tail's launch walks the binary
nodes whatever the layout is; after staged depths over the 4-wide nodes its
frames must equal the staged ones bit for bit, with and without shadow rays."""
import numpy as np
import pytest

from wavefrontpathtracing_gb300 import Renderer, scenes
from tests.helpers import load_scene_into

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nee", [0, 1])
@pytest.mark.parametrize("layout", [0, 1, 2])
def test_tail_equals_staged_depths(layout, nee):
    desc = scenes.mixed_box_scene(193, 141)
    kw = dict(max_bounces=7, spp=4, nee=nee, rr_start_depth=3, frame_seed=5, accumulate=False)
    with Renderer(193, 141, blas_layout=layout) as r:
        load_scene_into(r, desc)
        images, stats = [], []
        for tail in (0, 0, 60_000, 100_000):
            r.render(tail_paths=tail, **kw)
            images.append(r.read_image())
            stats.append(r.stats())
    assert stats[0]["tail_depth"] == 0 and 0 < stats[3]["tail_depth"] <= stats[2]["tail_depth"]
    for k in (1, 2, 3):
        assert np.array_equal(images[0].view(np.uint32), images[k].view(np.uint32))
        assert stats[0]["extend_rays_depth"] == stats[k]["extend_rays_depth"]
        assert stats[0]["shadow_rays_depth"] == stats[k]["shadow_rays_depth"]
