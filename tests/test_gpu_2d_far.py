"""2D nearest and silhouette searches where float rounding is of the size of the boxes' 1e-3
margin: scenes far from the origin or with large coordinates, and queries far from the
scene. Segments that share a vertex are at equal distances there as a rule, and the answer
is the reference's: the last one that its stack order visits, in every form of the search."""
import numpy as np
import pytest

from test_gpu_2d import close_frac
from test_gpu_parity import bits

pytestmark = pytest.mark.gpu


def loops(count, scale, shift, rng):
    """Noisy closed loops and open polylines over `scale` x `scale`, at `shift`."""
    verts, segs, off = [], [], 0
    for k in range(count):
        m = int(rng.integers(8, 200))
        c = rng.random(2)
        a = np.sort(rng.random(m)) * 2 * np.pi
        r = rng.uniform(0.01, 0.1) * (1 + 0.02 * rng.standard_normal(m))
        verts.append(np.stack([c[0] + r * np.cos(a), c[1] + r * np.sin(a)], 1))
        i = np.arange(m)
        segs.append(np.stack([i, (i + 1) % m], 1)[: m if k % 3 else m - 1] + off)
        off += m
    return (np.concatenate(verts) * scale + shift).astype(np.float32), np.concatenate(segs).astype(np.int32)


# (extent, shift of the scene, distance of the queries): at home, on either side of the
# coordinates from which the margin no longer covers the rounding, and far beyond
PLACES = [(20, 0, 0), (500, 0, 0), (1500, 0, 0), (4000, 0, 0), (8500, 0, 0), (20, 1700, 0), (20, 3e4, 0),
          (20, 1e5, 0), (20, 0, 1e4), (20, 0, 1e5), (1, 1e6, 1e6), (1e5, 0, 0), (3e19, 0, 0)]


@pytest.mark.parametrize("extent,shift,away", PLACES)
def test_far_answers_are_the_references(oracle_mod, extent, shift, away):
    import snch_lbvh_gb300 as snch
    rng = np.random.default_rng(5)
    v, sg = loops(60, extent, shift, rng)
    n = 140_000
    d = rng.random((n, 2)) * 1.2 - 0.1
    a = rng.random(n) * 2 * np.pi
    p = (d * extent + shift + away * np.stack([np.cos(a), np.sin(a)], 1)).astype(np.float32)
    p[:1000] = v[rng.integers(0, len(v), 1000)]
    flip = (rng.random(n) < 0.5).astype(np.uint8)
    s = snch.Scene2(v, sg)
    s.build()
    orc = oracle_mod.Tree2(v, sg)
    e = s.export()
    np.testing.assert_array_equal(e["nodes"], orc.nodes)
    orc.cones[:] = e["cones"]  # the tree's own: libm's acosf differs from CUDA's in a few of them
    oi, od = orc.nearest(p[:20_000])
    osd, osv = orc.silhouette(p[:20_000], flip[:20_000])
    first = None
    # a warp each, lanes and then warps (silhouettes), a lane each
    for m in (1, 20_000, 60_000, n):
        k = min(m, 20_000)
        i, dist = (x.cpu().numpy() for x in s.query_nearest(p[:m]))
        np.testing.assert_array_equal(bits(dist[:k]), bits(od[:k]))
        np.testing.assert_array_equal(i[:k].view(np.uint32), oi[:k])
        sd, sv = (x.cpu().numpy() for x in s.query_silhouette(p[:m], flip[:m]))
        if m > 1:
            # the cone test's acosf and atan2f are CUDA's, so not every one; but where the
            # distance is the oracle's, so is the vertex
            assert close_frac(sd[:k], osd) >= 0.999
            same = bits(sd[:k]) == bits(osd)
            assert (sv[:k][same] == osv[same]).mean() >= 0.9999
        got = i, bits(dist), bits(sd), sv
        for x, y in zip(first or (), got):  # the shorter batch again, in another form
            np.testing.assert_array_equal(x, y[: len(x)])
        first = got
    assert s.device_status() == 0


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 3e38])
def test_points_that_are_no_place(oracle_mod, bad):
    """NaN, infinite and huge coordinates: the oracle's answers, in each form."""
    import snch_lbvh_gb300 as snch
    rng = np.random.default_rng(6)
    v, sg = loops(20, 10, 0, rng)
    n = 30_000
    p = (rng.random((n, 2)) * 10).astype(np.float32)
    p[::7, 0] = bad
    p[::11, 1] = bad
    s = snch.Scene2(v, sg)
    s.build()
    orc = oracle_mod.Tree2(v, sg)
    oi, od = orc.nearest(p)
    osd, _ = orc.silhouette(p)
    for m in (20_000, n):
        i, dist = (x.cpu().numpy() for x in s.query_nearest(p[:m]))
        np.testing.assert_array_equal(i.view(np.uint32), oi[:m])
        np.testing.assert_array_equal(np.isnan(dist), np.isnan(od[:m]))
        ok = ~np.isnan(dist)
        np.testing.assert_array_equal(bits(dist[ok]), bits(od[:m][ok]))
        sd, _ = (x.cpu().numpy() for x in s.query_silhouette(p[:m]))
        assert close_frac(np.nan_to_num(sd, nan=-1.0), np.nan_to_num(osd[:m], nan=-1.0)) >= 0.999
    assert s.device_status() == 0
