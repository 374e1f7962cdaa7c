"""Topology and tree at the edges of the build kernels, against the oracle, bit for bit:
triangle counts around the 256-leaf blocks of the refit and the words and tiles of the edge
scan; a fan whose centre takes every probe of its place in the edge table, separate
triangles (every edge distinct), more vertices than table slots, degenerate triangles; the
view's objects."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import bits, check_cones, check_tri_ids

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def snch():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import snch_lbvh_gb300
    return snch_lbvh_gb300


def grid(n, rng):
    """n triangles of a noisy height field, numbered along its rows."""
    side = int(np.ceil(np.sqrt(n / 2))) + 1
    x, y = np.meshgrid(np.arange(side), np.arange(side), indexing="ij")
    v = np.stack([x.ravel(), y.ravel(), 0.3 * rng.standard_normal(side * side)], 1).astype(np.float32)
    q = (np.arange(side - 1)[:, None] * side + np.arange(side - 1)[None, :]).ravel()
    f = np.stack([np.stack([q, q + side, q + 1], 1), np.stack([q + 1, q + side, q + side + 1], 1)], 1).reshape(-1, 3)
    return v, f[:n].astype(np.int32)


def fan(n, rng):
    a = np.linspace(0, 6, n + 1)
    v = np.concatenate([[[0, 0, 0]], np.stack([np.cos(a), np.sin(a), 0.1 * rng.standard_normal(n + 1)], 1)])
    i = np.arange(1, n + 1)
    return v.astype(np.float32), np.stack([np.zeros(n, int), i, i + 1], 1).astype(np.int32)


def soup(n, rng):
    v = rng.random((3 * n, 3)) * 0.05 + np.repeat(rng.random((n, 3)), 3, 0)
    return v.astype(np.float32), np.arange(3 * n).reshape(n, 3).astype(np.int32)


def two_levels(n, rng):
    """Edges that all have their smaller vertex among the first few (an icosphere's coarse
    vertices come first), half of the triangles missing: those vertices' places overflow."""
    from snch_lbvh_gb300 import meshes
    v, f, _ = meshes.icosphere(4)
    return v.astype(np.float32), f[rng.permutation(len(f))[:n]]


def sparse(n, rng):
    """A height field whose vertices are spread over many unused ones."""
    v, f = grid(n, rng)
    big = np.zeros((len(v) * 50, 3), np.float32)
    big[::50] = v
    return big, (f * 50).astype(np.int32)


def degenerate(n, rng):
    v, f = grid(n, rng)
    f[::3, 1] = f[::3, 0]
    f[1::3] = f[1]
    return v, f


def device_words(ptr, rows, words):
    import torch

    class M:
        __cuda_array_interface__ = {"shape": (rows, words), "typestr": "<i4", "data": (int(ptr), False), "version": 3}
    return torch.as_tensor(M(), device="cuda").cpu().numpy()


CASES = [(grid, n) for n in (1, 2, 3, 255, 256, 257, 511, 512, 513, 1365, 1366, 43_691, 100_000)] + \
        [(fan, 5000), (fan, 200_000), (soup, 3000), (two_levels, 2560), (sparse, 700), (degenerate, 900)]


@pytest.mark.parametrize("make,n", CASES, ids=[f"{m.__name__}-{n}" for m, n in CASES])
def test_topology_and_tree(snch, oracle_mod, make, n):
    import torch
    rng = np.random.default_rng(n)
    v, f = make(n, rng)
    orc = oracle_mod.Tree(v, f)
    s = snch.Scene(v, f)
    s.compute_silhouettes()
    for _ in range(2):  # a second build over the same arrays
        s.build_bvh()
        te, to, ev = s.export_topology()
        np.testing.assert_array_equal(te, orc.tri_edges)
        np.testing.assert_array_equal(to, orc.tri_owned)
        np.testing.assert_array_equal(ev, orc.edge_verts)
        t = s.export_tree()
        np.testing.assert_array_equal(t["nodes"], orc.nodes)
        np.testing.assert_array_equal(bits(t["aabbs"]), bits(orc.aabbs))
        check_cones(t["cones"], orc.cones, orc.nodes, orc.d1)
        np.testing.assert_array_equal(s.leaf_ranks(), orc.leaf_ranks())
    assert s.device_status() == 0
    # the traversal records: child ids, rank and owned-edge count of leaf children, and
    # whether an internal child's cone test is settled
    if n > 1:
        t_ = len(f)
        rec = device_words(s.get_traversal_view().inner, t_ - 1, 16).view(np.uint32)
        np.testing.assert_array_equal(rec[:, 12:14], orc.nodes[: t_ - 1, 1:3])
        owned = (orc.tri_owned[orc.sorted_idx] >= 0).sum(1).astype(np.uint32)
        info = (orc.leaf_ranks() | owned << 30).astype(np.uint32)
        child = rec[:, 12:14].astype(np.int64) - (t_ - 1)
        half = t["cones"][orc.nodes[: t_ - 1, 1:3], 3]  # the built tree's own half angles
        settled = np.where(half >= np.float32(np.pi / 2), 1, np.where(half < 0, 2, 0))
        np.testing.assert_array_equal(rec[:, 14:16], np.where(child >= 0, info[child.clip(0)], settled))
        np.testing.assert_array_equal(rec[:, :12], bits(orc.aabbs)[orc.nodes[: t_ - 1, 1:3]].reshape(-1, 12))
    # near-first against the reference's order (ids up to the documented exact ties)
    p = torch.from_numpy((rng.random((2000, 3)) * (v.max(0) - v.min(0) + 0.1) + v.min(0)).astype(np.float32)).cuda()
    a = s.query_nearest(p) + s.query_silhouette(p)
    s.set_traversal(snch.TRAVERSAL_REFERENCE_ORDER)
    b = s.query_nearest(p) + s.query_silhouette(p)
    a, b, pts = [x.cpu().numpy() for x in a], [x.cpu().numpy() for x in b], p.cpu().numpy()
    np.testing.assert_array_equal(bits(a[1]), bits(b[1]))
    np.testing.assert_array_equal(bits(a[2]), bits(b[2]))
    check_tri_ids(a[0], b[0], b[1], pts, v, f)


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 1000])
def test_view_objects(snch, oracle_mod, n):
    """The objects of the byte-compatible view, and that a rebuild keeps them."""
    v, f = grid(n, np.random.default_rng(n))
    orc = oracle_mod.Tree(v, f)
    s = snch.Scene(v, f)
    s.compute_silhouettes()
    s.build_bvh()
    s.build_bvh()
    view = s.get_bvh_device_ptr()

    o = device_words(view.objects, n, 10)
    np.testing.assert_array_equal(o[:, :3], f)
    np.testing.assert_array_equal(o[:, 3:6], orc.tri_owned)
    ptrs = o[:, 6:].copy().view(np.uint64)
    verts = C.c_void_p()
    snch.lib().snch_scene_vertices(s._h, C.byref(verts))
    assert (ptrs == ptrs[0]).all() and ptrs[0, 0] == verts.value
    e = device_words(int(ptrs[0, 1]), len(orc.edge_verts), 8)
    np.testing.assert_array_equal(e[:, :4], orc.edge_verts)
    assert (e[:, 4:6].copy().view(np.uint64) == verts.value).all()


@pytest.mark.parametrize("make", [grid, soup])
@pytest.mark.parametrize("n", [769, 1023, 1024, 1025])
def test_one_block_trees(snch, oracle_mod, make, n):
    """Trees that one block of the refit covers, and the first that it does not."""
    test_topology_and_tree(snch, oracle_mod, make, n)
