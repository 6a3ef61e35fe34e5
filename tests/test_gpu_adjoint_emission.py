"""GPU: the emitter's gradient over many paths whose terms cancel.

With one emitter and a black environment the image is linear in the emitter's
strength s, so d(loss)/ds = sum over the image of dloss * image / s, summed
here in double.  Both sides are sums of the same single-precision path terms.
With image gradients of random sign their rounding errors are independent: a
pixel's 64 additions leave 1.4e-7 of it (root mean square), a term's six
roundings 0.9e-7, so the sums differ by 1.7e-7 of the root of the pixels'
squared terms; six times that is allowed.  A single-precision sum over the
16.8M paths is several times further off."""
import numpy as np
import pytest

from wavefrontpathtracing_gb300 import Renderer, scenes
from tests.helpers import load_scene_into

pytestmark = pytest.mark.gpu

SIDE = 512


@pytest.fixture(scope="module")
def room():
    desc = scenes.box_scene(SIDE, SIDE, subdivision=5)
    with Renderer(SIDE, SIDE) as r:
        load_scene_into(r, desc)
        yield r, desc


@pytest.mark.parametrize("nee,spp,seeds", [(0, 64, range(1, 9)), (1, 16, range(1, 3))])
def test_emitter_gradient_equals_the_double_sum_over_the_image(room, nee, spp, seeds):
    r, desc = room
    light = len(desc.instances) - 1
    strength = float(desc.instances[light][2]["base"]["emissive_strength"])
    for seed in seeds:
        rng = np.random.default_rng(seed)
        r.set_albedo(rng.uniform(0.1, 0.9, size=(r.scene_triangle_count(), 3)))
        dloss = (rng.normal(size=(SIDE, SIDE, 3)) / SIDE ** 2).astype(np.float32)
        kw = dict(max_bounces=6, spp=spp, frame_seed=seed, nee=nee, rr_start_depth=99)
        _, emission = r.adjoint(dloss, **kw)
        r.render(accumulate=False, **kw)
        terms = dloss.astype(np.float64) * r.read_image()[..., :3] / strength
        assert abs(emission[light] - terms.sum()) <= 1e-6 * np.sqrt((terms ** 2).sum()), seed
        assert not np.any(emission[:light])


@pytest.mark.parametrize("nee", [0, 1])
def test_each_of_three_emitters_has_its_own_gradient(nee):
    """Paths meet several emitters, so their sums change emitter on the way.  No
    path depends on a strength, so the image with one strength doubled less the
    image is that emitter's part of it.  The difference of two images leaves
    sqrt(1 + 4) times one's rounding error of the whole image: 3.3e-7 of the
    root of the pixels' squared terms, six times that allowed."""
    side, spp, strengths = 256, 16, (15.0, 4.0, 40.0)
    desc = scenes.box_scene(side, side, subdivision=4)
    light = len(desc.instances) - 1
    _, _, m = desc.instances[light]
    for k, at in ((1, (0.3, -0.2, 0.1)), (2, (-0.3, -0.4, -0.2))):
        t = np.eye(4)
        t[:3, 3] = at
        extra = m.copy()
        extra["base"]["emissive_strength"] = strengths[k]
        desc.instances.append((desc.instances[light][0], t, extra))
    with Renderer(side, side) as r:
        load_scene_into(r, desc)
        rng = np.random.default_rng(7)
        r.set_albedo(rng.uniform(0.1, 0.9, size=(r.scene_triangle_count(), 3)))
        dloss = (rng.normal(size=(side, side, 3)) / side ** 2).astype(np.float32)
        kw = dict(max_bounces=6, spp=spp, frame_seed=5, nee=nee, rr_start_depth=99)

        def image():
            r.render(accumulate=False, **kw)
            return r.read_image()[..., :3].astype(np.float64)

        _, emission = r.adjoint(dloss, **kw)
        base = image()
        for k, s in enumerate(strengths):
            r.set_emission(light + k, 2.0 * s)
            part = image() - base
            r.set_emission(light + k, s)
            assert np.linalg.norm(part) > 1e-3 * np.linalg.norm(base)
            want, whole = (dloss * part).sum() / s, np.sqrt(((dloss * base) ** 2).sum()) / s
            assert abs(emission[light + k] - want) <= 2e-6 * whole, (k, emission, want, whole)
    assert not np.any(emission[:light])
