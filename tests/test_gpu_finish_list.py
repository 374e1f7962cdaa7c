"""Searches that one launch leaves to the next: a full list, a list of a few entries and none
(as without memory for it) give the one-query-per-lane answers; a captured batch, which has no
list, searches a warp each and not a lane each; ids are the same ones or exact ties."""
import numpy as np
import pytest

from test_gpu_parity import bits, built_scene, check_edge_ids, check_tri_ids

pytestmark = pytest.mark.gpu


def closed_mesh(n, seed=4):
    import snch_lbvh_gb300 as snch
    from snch_lbvh_gb300 import meshes
    v, f = meshes.noisy_icosphere(5, 1.0, 0.01, seed=0)
    s = built_scene(snch, v, f)
    rng = np.random.default_rng(seed)
    p = (rng.random((n, 3)) * 2.4 - 1.2).astype(np.float32)
    return s, v, f, p, (rng.random(n) < 0.5).astype(np.uint8)


def compare(s, v, f, p, got, exp):
    i, d, sd, se = ([x.cpu().numpy() for x in r] for r in zip(got, exp))
    np.testing.assert_array_equal(bits(d[0]), bits(d[1]))
    np.testing.assert_array_equal(bits(sd[0]), bits(sd[1]))
    check_tri_ids(i[0], i[1], d[1], p, v, f)
    check_edge_ids(se[0], se[1], sd[1], p, v, s.export_topology()[2])
    assert s.device_status() == 0


# one query per lane and then per warp; packets from the counter; packets from the pools
@pytest.mark.parametrize("n", [30_000, 140_011, 32 * 2**15 + 33])
@pytest.mark.parametrize("most", [0, 1, 33, 100, 5000])
def test_short_lists(n, most):
    import snch_lbvh_gb300 as snch
    s, v, f, p, flip = closed_mesh(n)

    def run():
        return s.query_nearest(p) + s.query_silhouette(p, flip)

    s.set_option(snch.OPT_PACKET, 0)
    exp = run()
    s.set_option(snch.OPT_PACKET, 2)
    s.set_option(snch.OPT_FINISH_LIST, most)
    assert s.get_option(snch.OPT_FINISH_LIST) == most
    compare(s, v, f, p, run(), exp)


@pytest.mark.parametrize("most", [0, 33])
def test_short_lists_of_batched_and_seeded_queries(most):
    import snch_lbvh_gb300 as snch
    import torch
    s, v, f, p, flip = closed_mesh(150_000)
    b = snch.BatchedScene([(v, f), (v * np.float32(0.5), f)])
    b.compute_silhouettes()
    b.build_bvh()
    m = torch.from_numpy((np.arange(len(p)) % 2).astype(np.int32)).cuda()
    out = []
    for packet, k in ((0, -1), (2, most)):
        for x in (s, b):
            x.set_option(snch.OPT_PACKET, packet)
            x.set_option(snch.OPT_FINISH_LIST, k)
        i, d = s.query_nearest(p)
        r = (d * torch.from_numpy(np.random.default_rng(1).choice([0.5, 2.0], len(p)).astype(np.float32)).cuda())
        out.append((s.query_nearest_seeded(p, r), s.query_silhouette_seeded(p, r, flip),
                    b.query_nearest_batch(m, p), b.query_silhouette_batch(m, p, flip)))
    for x, y in zip(*out):
        for a, c in zip(x, y):
            if a.dtype == torch.float32:
                assert torch.equal(a.view(torch.int32), c.view(torch.int32))
            else:  # ids: exact ties apart
                assert int((a != c).sum()) <= 15
    assert s.device_status() == 0 and b.device_status() == 0


def test_options_limits():
    import snch_lbvh_gb300 as snch
    s = closed_mesh(1)[0]
    with pytest.raises(snch.SnchError):
        s.set_option(snch.OPT_FINISH_LIST, -2)


@pytest.mark.parametrize("n", [30_000, 65_000, 100_000])
def test_captured_batches(n):
    """The captured answers, and that an unordered batch (below 65,536) is not searched a lane
    each: 10 to 12 ms there, about a millisecond with a warp each."""
    import snch_lbvh_gb300 as snch
    import torch
    s, v, f, p, flip = closed_mesh(n)
    p, flip = torch.from_numpy(p).cuda(), torch.from_numpy(flip).cuda()

    def run():
        st = torch.cuda.current_stream()
        return s.query_nearest(p, stream=st) + s.query_silhouette(p, flip, stream=st)

    def captured():
        run()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            out = run()
        t = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        ms = []
        for _ in range(4):
            t[0].record()
            g.replay()
            t[1].record()
            t[1].synchronize()
            ms.append(t[0].elapsed_time(t[1]))
        return out, min(ms)

    s.set_option(snch.OPT_PACKET, 0)
    exp, lanes = captured()
    s.set_option(snch.OPT_PACKET, 2)
    got, own = captured()
    compare(s, v, f, p.cpu().numpy(), got, exp)
    assert own < 0.5 * lanes, (own, lanes)


@pytest.mark.parametrize("n", [131_073, 149_440, 149_441])
def test_sparse_silhouette_ids(n):
    """Lanes first on a sparse batch: every edge id is the per-lane search's, or an exact tie."""
    import snch_lbvh_gb300 as snch
    from snch_lbvh_gb300 import meshes
    v, f = meshes.torus(0.8, 0.3, 1868, 320)[:2]
    v = v.astype(np.float32)
    s = built_scene(snch, v, f)
    rng = np.random.default_rng(n)
    p = (rng.random((n, 3)) * 2.4 - 1.2).astype(np.float32)
    flip = (rng.random(n) < 0.5).astype(np.uint8)
    d, e = (x.cpu().numpy() for x in s.query_silhouette(p, flip))
    s.set_option(snch.OPT_PACKET, 0)
    d0, e0 = (x.cpu().numpy() for x in s.query_silhouette(p, flip))
    np.testing.assert_array_equal(bits(d), bits(d0))
    check_edge_ids(e, e0, d0, p, v, s.export_topology()[2])
    assert s.device_status() == 0


@pytest.mark.parametrize("n", [320 * 192 - 1, 65_535, 65_536, 131_073])
def test_crowded_silhouette_batches(n):
    """Around the size at which an ordered batch of a small mesh runs as packets."""
    import snch_lbvh_gb300 as snch
    from snch_lbvh_gb300 import meshes
    v, f = meshes.noisy_icosphere(2, 1.0, 0.01, seed=0)
    s = built_scene(snch, v, f)
    rng = np.random.default_rng(n)
    p = (rng.random((n, 3)) * 2.4 - 1.2).astype(np.float32)
    flip = (rng.random(n) < 0.5).astype(np.uint8)
    got = s.query_nearest(p) + s.query_silhouette(p, flip)
    s.set_option(snch.OPT_PACKET, 0)
    compare(s, v, f, p, got, s.query_nearest(p) + s.query_silhouette(p, flip))
