"""Small builds sort by rank (scan_sort.cu rank_sort_kernel): the stable order of the
Morton codes, equal codes included, at the edges of its warps and chunks and of its range.
Query batches around the sizes up to which a shorter key orders them: the answers of the
same batch in input order."""
import numpy as np
import pytest

from test_gpu_parity import bits, built_scene, check_edge_ids, check_tri_ids

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 32, 33, 127, 128, 129, 255, 257, 1000, 4097, 12288, 12289]


def check_order(idx, code, n):
    assert np.array_equal(np.sort(idx), np.arange(n))
    by_input = np.empty(n, np.uint32)
    by_input[idx] = code
    np.testing.assert_array_equal(idx, np.argsort(by_input, kind="stable"))


@pytest.mark.parametrize("n", SIZES)
def test_order_of_small_builds(oracle_mod, n):
    import snch_lbvh_gb300 as snch
    rng = np.random.default_rng(n)
    # a third of the triangles repeat others, so codes repeat near and far apart
    c = rng.random((n, 3))
    c[rng.random(n) < 0.33] = c[: max(1, n // 50)][rng.integers(0, max(1, n // 50), 1)[0]]
    v = (c[:, None, :] + 0.01 * np.eye(3)[None]).reshape(-1, 3).astype(np.float32)
    f = np.arange(3 * n, dtype=np.int32).reshape(-1, 3)
    s = snch.Scene(v, f)
    s.compute_silhouettes()
    for _ in range(2):
        s.build_bvh()
        t = s.export_tree()
        check_order(t["sorted_idx"], t["morton"], n)
    orc = oracle_mod.Tree(v, f)
    np.testing.assert_array_equal(t["sorted_idx"], orc.sorted_idx)
    np.testing.assert_array_equal(t["morton"], orc.morton[orc.sorted_idx])
    assert s.device_status() == 0
    s2 = snch.Scene2(np.ascontiguousarray(v[:, :2]), f[:, :2].copy())
    s2.build()
    e = s2.export()
    check_order(e["sorted_idx"], e["morton"], n)


@pytest.mark.parametrize("order_bits", [12, 24, 30])
@pytest.mark.parametrize("n", [65536, 1 << 17, (1 << 17) + 1, 1 << 22, (1 << 22) + 1])
def test_ordered_batches_answer_alike(n, order_bits):
    import snch_lbvh_gb300 as snch
    import torch
    from snch_lbvh_gb300 import meshes
    v, f = meshes.noisy_icosphere(3, 1.0, 0.01, seed=0)
    s = built_scene(snch, v, f)
    s.set_option(snch.OPT_ORDER_BITS, order_bits)
    g = torch.Generator(device="cuda").manual_seed(n)
    p = 2.4 * torch.rand(n, 3, generator=g, device="cuda") - 1.2
    d = torch.randn(n, 3, generator=g, device="cuda")
    tmax = torch.rand(n, generator=g, device="cuda") * 2.0
    q = p[: (1 << 17) + 1]

    def everything():
        out = s.query_ray(p, d, tmax)
        if n <= len(q):
            out += s.query_nearest(q) + s.query_silhouette(q)
        return [x.cpu().numpy() for x in out]

    a = everything()
    s.set_option(snch.OPT_QUERY_ORDER, 0)
    b = everything()
    for k, (x, y) in enumerate(zip(a, b)):
        if k not in (4, 7):  # ids: up to the documented exact ties
            np.testing.assert_array_equal(bits(x) if x.dtype == np.float32 else x, bits(y) if y.dtype == np.float32 else y)
    if n <= len(q):
        check_tri_ids(a[4], b[4], b[5], q.cpu().numpy(), v, f)
        check_edge_ids(a[7], b[7], b[6], q.cpu().numpy(), v, s.export_topology()[2])
    assert s.device_status() == 0
