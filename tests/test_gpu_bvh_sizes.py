"""GPU: the BLAS builder at the edges of its phases — a lane per triangle (10 /
11, 32 / 33), a subtree's block (128 / 129), a chunk of the large phase (1,024
/ 1,025) — for few, odd and the most bins, with zero coordinates of both signs,
ties and large leaves that no plane splits, byte for byte against the oracle."""
import numpy as np
import pytest

from wavefrontpathtracing_gb300 import Renderer, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def r():
    with Renderer(8, 8) as rr:
        yield rr


@pytest.mark.parametrize("ic,single,max_leaf", [(2, 0, 0), (8, 0, 0), (33, 0, 2), (64, 1, 0)])
@pytest.mark.parametrize("n", [1, 2, 3, 9, 10, 11, 31, 32, 33, 127, 128, 129, 257, 1023, 1024, 1025, 2049, 4100])
def test_every_phase_boundary(orc, r, n, ic, single, max_leaf):
    tris = scenes.triangle_soup(n, seed=n, mu=-2.0)
    rng = np.random.default_rng(n)
    for v in ("v0", "v1", "v2"):
        p = tris[v]["position"]
        p -= np.float32(0.5)
        mask = rng.random(p.shape) < 0.2
        p[mask] = np.where(rng.random(mask.sum()) < 0.5, np.float32(-0.0), np.float32(0.0))
        if n % 2:
            p[:] = np.round(p * 8) / 8   # equal centroids and costs
    tris[: n // 3] = tris[0]   # a third of them one triangle: a leaf that no plane splits
    want = orc.bvh_build(tris, ic, bool(single), max_leaf)
    got = r.bvh_build(tris, ic, bool(single), max_leaf)
    assert np.array_equal(got, want)
