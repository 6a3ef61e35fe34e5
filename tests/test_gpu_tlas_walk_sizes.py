"""GPU: the agglomerative TLAS walk (tlas_metric 0 / 1) on both sides of every
size at which its launch takes another kernel (a warp of one or two list
positions per lane, blocks of 128 with 1 to 12 positions per thread, of 256
with 8 or 16, the scanning block), byte for byte against the oracle through
both entry points; and boxes of infinities and NaN, which have no order: the
walk ends with a tree that holds every instance once and every index in range."""
import ctypes

import numpy as np
import pytest

import wavefrontpathtracing_gb300 as wf
from tests.test_gpu_tlas_walk import lattice_instances, test_walk_equals_the_oracle_with_ties as walk_equals_the_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("n", [3, 63, 64, 66, 127, 128, 129, 192, 255, 256, 257, 385, 512, 513, 640, 768, 769, 1026, 1280,
                               1281, 1400, 1536, 1537, 3000])
def test_every_kernel_of_the_walk(orc, n, metric):
    walk_equals_the_oracle(orc, n, metric)


@pytest.mark.parametrize("metric", [0, 1])
@pytest.mark.parametrize("n", [2, 5, 40, 130, 300, 600, 1300, 1600, 4097])
def test_boxes_without_order_end_in_a_whole_tree(n, metric):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    inst = lattice_instances(n, seed=n)
    special = np.array([np.nan, np.inf, -np.inf, 3.4e38, -3.4e38, 0.0, 1.0], np.float32)
    for k in ("aabb_min", "aabb_max"):
        some = rng.random((n, 3)) < 0.3
        inst[k][some] = special[rng.integers(0, len(special), size=int(some.sum()))]
    with wf.Renderer(8, 8, tlas_metric=metric) as r:
        blob = r.tlas_build(inst)
    boxes = np.concatenate([inst["aabb_min"], inst["aabb_max"]], axis=1).astype(np.float32)
    d_boxes = torch.from_numpy(boxes.copy()).cuda()
    d_nodes = torch.zeros(16 * n, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    rc = wf.load().wf_tlas_build_noalloc(ctypes.c_void_p(d_boxes.data_ptr()), n, ctypes.c_void_p(d_nodes.data_ptr()),
                                         metric, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    nodes = blob[8:8 + 64 * n].view(np.uint32).reshape(2 * n, 8)
    assert np.array_equal(nodes, d_nodes.cpu().numpy().view(np.uint32).reshape(2 * n, 8))
    seen, todo = [], [0]
    while todo:
        k = todo.pop()
        word = int(nodes[k, 3])
        if word == 0:
            seen.append(int(nodes[k, 7]))
        else:
            assert 0 < word >> 16 < 2 * n and 0 < word & 0xFFFF < 2 * n and len(todo) < 2 * n
            todo += [word >> 16, word & 0xFFFF]
    assert sorted(seen) == list(range(n))
