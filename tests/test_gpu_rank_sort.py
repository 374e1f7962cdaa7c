"""Small builds sort by rank (scan_sort.cu rank_sort_kernel): the stable order of the
Morton codes, equal codes included, at the edges of its warps and chunks and of its range."""
import numpy as np
import pytest

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
