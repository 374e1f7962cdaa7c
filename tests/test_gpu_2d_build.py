"""2D builds at the edges of the build kernels' blocks, against the oracle bit for bit: scene
box (through the codes), tree, boxes, and the leaves' ranks, which decide between segments
that meet in the nearest vertex."""
import numpy as np
import pytest

from test_gpu_2d import check_cones2
from test_gpu_parity import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 127, 128, 129, 255, 256, 257, 12_288, 12_289, 70_001])
def test_tree_and_ranks(oracle_mod, n):
    import snch_lbvh_gb300 as snch
    rng = np.random.default_rng(n)
    a = np.sort(rng.random(n)) * 2 * np.pi
    r = 4.0 * (1 + 0.1 * rng.standard_normal(n))
    v = np.concatenate([np.stack([r * np.cos(a), r * np.sin(a)], 1), [[-9.0, 2.0]]]).astype(np.float32)
    i = np.arange(n)
    sg = np.stack([i, i + 1], 1).astype(np.int32)  # one open polyline; its last vertex is far out
    s = snch.Scene2(v, sg)
    orc = oracle_mod.Tree2(v, sg)
    p = np.concatenate([v, v * np.float32(1.5)])[:20_000]
    oi, od = orc.nearest(p)
    for _ in range(2):  # a second build over the same arrays
        s.build()
        e = s.export()
        np.testing.assert_array_equal(e["sorted_idx"], orc.sorted_idx)
        np.testing.assert_array_equal(e["nodes"], orc.nodes)
        np.testing.assert_array_equal(bits(e["aabbs"]), bits(orc.aabbs))
        check_cones2(e["cones"], orc.cones, orc.nodes, orc.d1)
        idx, dist = (x.cpu().numpy() for x in s.query_nearest(p))
        np.testing.assert_array_equal(bits(dist), bits(od))
        np.testing.assert_array_equal(idx.view(np.uint32), oi)
    assert s.device_status() == 0


def test_fast_cone_test_agrees_with_exact():
    """The 2D cone test's filter decides only where its error bound allows, and then as the
    exact test: 4M random cases, half of them within 1e-3 rad of the decision."""
    import ctypes as C

    import snch_lbvh_gb300 as snch
    import torch
    counts = torch.zeros(3, dtype=torch.int64, device="cuda")
    for seed in (1, 2):
        snch.check(snch.lib().snch_selfcheck_cone_filter2(2_000_000, seed, C.c_void_p(counts.data_ptr()),
                                                          C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    agree, disagree, undecided = (int(x) for x in counts.cpu())
    assert agree + disagree + undecided == 4_000_000
    assert disagree == 0
    assert agree >= 0.5 * 4_000_000, (agree, undecided)
