"""GPU: launches of every size relative to the traversal grid.

A warp's first rays are its own by its number, spread over the grid's warps
when the launch has fewer rays than the grid has lanes; later rays come from a
counter.  Sizes at and around the edges of that rule (one ray, a warp, the
grid's warps, its lanes) must give the oracle's hits bit for bit and write
nothing past the last ray.

Waves of at most 65,536 paths without shadow rays run whole in one launch;
their images and ray counts must equal the staged launches' (which profiled
frames use) and the megakernel's, below, at and above that size.

Shade places a block's continuation and shadow rays in the queues by octant:
around the block's size no ray may be lost or written twice, so images must
equal the megakernel's."""
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


# 65,535 / 65,536 / 65,538 paths; a wave split into short ones; many samples; no bounce
@pytest.mark.parametrize("width,height,spp,bounces,rr,wave", [
    (1, 1, 1, 4, 99, 0), (257, 255, 1, 2, 99, 0), (256, 256, 1, 4, 3, 0), (10923, 6, 1, 1, 99, 0),
    (97, 61, 5, 6, 2, 1000), (60, 40, 7, 0, 99, 0)])
def test_whole_waves_equal_staged_launches(width, height, spp, bounces, rr, wave):
    desc = scenes.mixed_box_scene(width, height)
    kw = dict(max_bounces=bounces, spp=spp, nee=0, rr_start_depth=rr, wave_paths=wave, frame_seed=5)
    with Renderer(width, height) as r:
        load_scene_into(r, desc)
        images, stats = [], []
        for extra in (dict(), dict(profile=True), dict(megakernel=True)):
            r.render(accumulate=False, **kw, **extra)
            r.render(accumulate=True, **kw, **extra)   # a second call on top
            images.append(r.read_image())
            stats.append(r.stats())
    assert width * height == 1 or bounces == 0 or images[0][..., :3].max() > 0.0   # the light is behind the camera
    for k in (1, 2):
        assert np.array_equal(images[0].view(np.uint32), images[k].view(np.uint32))
        assert stats[0]["rays_extend"] == stats[k]["rays_extend"] and stats[0]["rays_connect"] == 0
    assert stats[0]["extend_rays_depth"] == stats[1]["extend_rays_depth"]
    assert (stats[0]["launches"] < stats[1]["launches"]) == ((wave or width * height * spp) <= 65536)


@pytest.mark.parametrize("width,height,spp,bounces,wave", [
    (1, 1, 1, 3, 0), (127, 1, 1, 3, 0), (128, 1, 1, 3, 0), (43, 1, 3, 3, 0), (61, 37, 2, 6, 0), (61, 37, 2, 6, 257),
    (641, 359, 1, 2, 0)])
def test_queues_hold_every_ray(width, height, spp, bounces, wave):
    desc = scenes.mixed_box_scene(width, height)
    kw = dict(max_bounces=bounces, spp=spp, nee=1, rr_start_depth=2, wave_paths=wave, frame_seed=11, accumulate=False)
    with Renderer(width, height) as r:
        load_scene_into(r, desc)
        r.render(**kw)
        image = r.read_image()
        r.render(megakernel=True, **kw)
        assert np.array_equal(image.view(np.uint32), r.read_image().view(np.uint32))
