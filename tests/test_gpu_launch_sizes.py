"""GPU: launches of every size relative to the traversal grid.

A warp's first rays are its own by its number, spread over the grid's warps
when the launch has fewer rays than the grid has lanes; later rays come from a
counter.  Sizes at and around the edges of that rule (one ray, a warp, the
grid's warps, its lanes) must give the oracle's hits bit for bit and write
nothing past the last ray."""
import numpy as np
import pytest

from wavefrontpathtracing_gb300 import Renderer, scenes
from tests.helpers import load_scene_into, oracle_scene_from_renderer
from tests.test_gpu_trace import assert_hits_equal, random_rays

pytestmark = pytest.mark.gpu

GUARD = 0x5A5A5A5A


@pytest.fixture(scope="module")
def scene(orc):
    desc = scenes.instanced_scene(width=16, height=16, instances=24, freqs=(4, 6))
    with Renderer(16, 16) as r:
        ids = load_scene_into(r, desc)
        sc, _ = oracle_scene_from_renderer(orc, desc, r, ids)
        rays = random_rays(180_001, 0.0, 100.0, seed=9)
        yield r, rays, {f: sc.trace(rays, flags=f, threads=8)[0] for f in (0, 1)}


# 152 SMs x 9 blocks x 4 warps = 5,472 warps, 175,104 lanes
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 5471, 5472, 5473, 10_945, 175_103, 175_104, 175_105, 180_001])
@pytest.mark.parametrize("any_hit", [False, True])
def test_every_launch_size_gives_the_oracle_hits(scene, n, any_hit):
    torch = pytest.importorskip("torch")
    r, rays, want = scene
    d_rays = torch.from_numpy(rays[:n].view(np.float32).reshape(n, 8).copy()).cuda()
    d_hits = torch.full((n + 64, 5), GUARD, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    r.trace_device(d_rays.data_ptr(), n, d_hits.data_ptr(), any_hit=any_hit)
    r.synchronize()
    got = d_hits.cpu().numpy()
    assert (got[n:] == GUARD).all()
    assert_hits_equal(got[:n].copy().view(want[0].dtype).reshape(n), want[int(any_hit)][:n], f"{n} rays")
