"""GPU: the agglomerative TLAS walk (tlas_metric 0 / 1) at the edges of its
block: a warp, one / two / four list positions per thread in registers, the
positions past them, the list in shared memory (7,168) and beyond.  Boxes on a
coarse lattice with duplicates and flat boxes make most pairing values equal,
so the lowest-position rule decides almost every match; the blobs must equal
the oracle's byte for byte, through both entry points."""
import ctypes

import numpy as np
import pytest

import wavefrontpathtracing_gb300 as wf
from wavefrontpathtracing_gb300.abi import bvh_instance_dtype

pytestmark = pytest.mark.gpu


def lattice_instances(n, seed):
    rng = np.random.default_rng(seed)
    inst = np.zeros(n, dtype=bvh_instance_dtype)
    lo = rng.integers(-3, 4, size=(n, 3)).astype(np.float32)
    inst["aabb_min"] = lo
    inst["aabb_max"] = lo + rng.integers(0, 3, size=(n, 3)).astype(np.float32)
    inst["aabb_min"][n // 2] *= np.float32(-0.0)   # signed zeros
    inst["aabb_max"][n // 2] = 0.0
    return inst


@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 65, 1023, 1024, 1025, 2048, 2049, 4096, 4097, 7168, 7169])
def test_walk_equals_the_oracle_with_ties(orc, n, metric):
    torch = pytest.importorskip("torch")
    inst = lattice_instances(n, seed=n)
    want = orc.tlas_build(inst, metric=metric)
    with wf.Renderer(8, 8, tlas_metric=metric) as r:
        assert np.array_equal(r.tlas_build(inst), want)
    boxes = np.concatenate([inst["aabb_min"], inst["aabb_max"]], axis=1).astype(np.float32)
    d_boxes = torch.from_numpy(boxes.copy()).cuda()
    d_nodes = torch.full((16 * n + 16,), -1.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    rc = wf.load().wf_tlas_build_noalloc(ctypes.c_void_p(d_boxes.data_ptr()), n, ctypes.c_void_p(d_nodes.data_ptr()),
                                         metric, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0, wf.load().wf_last_error()
    torch.cuda.synchronize()
    got = d_nodes.cpu().numpy()
    assert (got[16 * n:] == -1.0).all()
    if n > 1:   # the second node slot of a single instance is written by no build
        assert np.array_equal(got[:16 * n].view(np.uint8), want[8:8 + 64 * n])
