"""Small batches run one query per warp, and the last long packets of a larger batch
finish that way: the answers equal the one-query-per-lane searches bit for bit (the
same minimum over the same leaves, ties by rank), at the edges of the size rules, on
meshes from one triangle up, inside closed meshes, seeded, and in batched scenes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def snch():
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import snch_lbvh_gb300
    return snch_lbvh_gb300


def mesh(level):
    from snch_lbvh_gb300 import meshes
    if level >= 0:
        return meshes.noisy_icosphere(level, 1.0, 0.01, seed=level + 1)
    v = np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0], [1, 1, 0.5]], np.float32)
    return v, np.array([[0, 1, 2], [1, 3, 2]], np.int32)[:-level]  # -1: one triangle, -2: two


def scene(snch, level):
    s = snch.Scene(*mesh(level))
    s.compute_silhouettes()
    s.build_bvh()
    return s


def points(n, seed=0):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return ((2 * torch.rand(n, 3, generator=g, device="cuda") - 1) * 1.2,
            (torch.rand(n, generator=g, device="cuda") < 0.5).to(torch.uint8))


def both_forms(snch, s, run):
    """run() with one query per lane, then with the form left to the library."""
    s.set_option(snch.OPT_PACKET, 0)
    a = run()
    s.set_option(snch.OPT_PACKET, 2)
    b = run()
    assert s.device_status() == 0
    return a, b


def same(a, b):
    import torch
    for x, y in zip(a, b):
        assert torch.equal(x.view(torch.int32), y.view(torch.int32)), int((x != y).sum())


@pytest.mark.parametrize("level", [-1, -2, 0, 2, 4])
@pytest.mark.parametrize("n", [1, 2, 3, 31, 1000])
def test_small_batches(snch, level, n):
    s = scene(snch, level)
    p, f = points(n, seed=n)
    same(*both_forms(snch, s, lambda: s.query_nearest(p) + s.query_silhouette(p, f)))


# around the sizes where the lanes take the short searches first (24,576), where a
# batch is ordered (65,536), where nearest (98,304) and
# silhouette (131,072) batches become packets, and where packets draw from the
# per-SM pools (2^15 packets), closed mesh: packets of thousands of steps
@pytest.mark.parametrize("n", [24_576, 24_577, 65_535, 65_536, 98_304, 98_305, 131_072, 131_073, 32 * 2**15 - 31, 32 * 2**15 + 1])
def test_size_rules_on_a_closed_mesh(snch, n):
    s = scene(snch, 5)
    p, f = points(n, seed=7)
    same(*both_forms(snch, s, lambda: s.query_nearest(p) + s.query_silhouette(p, f)))


@pytest.mark.parametrize("n", [5000, 30_000])
def test_seeded_small_batches(snch, n):
    import torch
    s = scene(snch, 4)
    p, f = points(n, seed=3)
    i, d = s.query_nearest(p)
    sd, e = s.query_silhouette(p, f)
    for scale in (0.5, 1.0, 2.0):  # below, at and above the answers
        rn = torch.nextafter(d * scale, torch.full_like(d, float("inf")))
        rs = torch.nextafter(sd * scale, torch.full_like(sd, float("inf")))
        a, b = both_forms(snch, s, lambda: s.query_nearest_seeded(p, rn) + s.query_silhouette_seeded(p, rs, f))
        same(a, b)
        same(b, (i, d, sd, e))


@pytest.mark.parametrize("n", [777, 30_001, 200_000])
def test_batched_scene(snch, n):
    import torch
    meshes = [mesh(k) for k in (-1, 3, 5, -2)] + [(np.zeros((0, 3), np.float32), np.zeros((0, 3), np.int32))]
    s = snch.BatchedScene(meshes)
    s.compute_silhouettes()
    s.build_bvh()
    p, f = points(n, seed=5)
    m = torch.randint(0, len(meshes), (n,), generator=torch.Generator().manual_seed(1), dtype=torch.int32).cuda()
    same(*both_forms(snch, s, lambda: s.query_nearest_batch(m, p) + s.query_silhouette_batch(m, p, f)))


@pytest.mark.parametrize("segments", [2, 3, 40, 20_000])
@pytest.mark.parametrize("n", [1, 24_576, 24_577, 131_072, 131_073])
def test_2d_forms_agree(segments, n):
    """A warp per query, lanes then warps, and a lane per query: one batch of n queries
    against the same queries in batches of 1,000 (a warp each), bit for bit (2D boxes are
    inflated, so the bound never cuts off an equal candidate)."""
    import snch_lbvh_gb300 as snch
    import torch
    rng = np.random.default_rng(segments)
    k = segments
    a = np.sort(rng.random(k)) * 2 * np.pi
    r = 5.0 * (1 + 0.05 * rng.standard_normal(k))
    v = np.stack([r * np.cos(a), r * np.sin(a)], 1).astype(np.float32)
    i = np.arange(k)
    sg = np.stack([i, (i + 1) % k], 1)[: k if k > 2 else k - 1].astype(np.int32)
    sg = np.concatenate([sg, sg[:1]]) if k == 2 else sg
    s = snch.Scene2(v, sg)
    s.build()
    p = ((rng.random((n, 2)) - 0.5) * 14).astype(np.float32)
    p[: min(n, k)] = v[: min(n, k)]  # on vertices: distance 0 and ties of two segments
    p, flip = torch.from_numpy(p).cuda(), torch.from_numpy((rng.random(n) < 0.5).astype(np.uint8)).cuda()
    part = slice(max(0, n - 1000), n), slice(0, min(n, 1000))
    idx, dist = s.query_nearest(p)
    sd, sv = s.query_silhouette(p, flip)
    for w in part:
        bi, bd = s.query_nearest(p[w].contiguous())
        bsd, bsv = s.query_silhouette(p[w].contiguous(), flip[w].contiguous())
        assert torch.equal(dist[w].view(torch.int32), bd.view(torch.int32))
        assert torch.equal(sd[w].view(torch.int32), bsd.view(torch.int32))
        assert torch.equal(idx[w], bi)
        assert torch.equal(sv[w], bsv)
    assert s.device_status() == 0


@pytest.mark.parametrize("n", [30_000, 100_000])
def test_forms_under_capture(snch, n):
    """A captured batch of a size that would be finished by a second launch: the replayed
    answers are the direct ones, bit for bit, and ids up to exact ties at distance equal."""
    import torch
    v, f = mesh(3)
    s = snch.Scene(v, f)
    s.compute_silhouettes()
    s.build_bvh()
    p, flip = points(n, seed=8)
    a = np.linspace(0, 2 * np.pi, 500, endpoint=False)
    s2 = snch.Scene2(np.stack([np.cos(a), np.sin(a)], 1).astype(np.float32) * (1 + 0.01 * np.sin(40 * a))[:, None].astype(np.float32),
                     np.stack([np.arange(500), (np.arange(500) + 1) % 500], 1).astype(np.int32))
    s2.build()
    p2 = p[:, :2].contiguous()

    def everything():
        st = torch.cuda.current_stream()
        return (s.query_nearest(p, stream=st) + s.query_silhouette(p, flip, stream=st) +
                s2.query_nearest(p2, stream=st) + s2.query_silhouette(p2, flip, stream=st))

    direct = [x.clone() for x in everything()]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = everything()
    for x in out:
        x.zero_()
    g.replay()
    torch.cuda.synchronize()
    for k in (1, 2, 5, 6):  # distances
        assert torch.equal(out[k].view(torch.int32), direct[k].view(torch.int32)), k
    for k in (0, 3, 4, 7):
        assert (out[k] == direct[k]).float().mean().item() > 0.999, k
    assert s.device_status() == 0 and s2.device_status() == 0


@pytest.mark.parametrize("n", [131_073, 149_440, 149_441])
def test_sparse_silhouette_batches(snch, n):
    """Around the sizes at which a batch is sparse enough for lanes and then warps: the
    one-query-per-lane answers, bit for bit, ids up to exact ties."""
    import torch
    from snch_lbvh_gb300 import meshes
    v, f = meshes.torus(0.8, 0.3, 1868, 320)[:2]
    assert len(f) == 8 * 149_440
    s = snch.Scene(v.astype(np.float32), f)
    s.compute_silhouettes()
    s.build_bvh()
    p, flip = points(n, seed=3)
    a = s.query_silhouette(p, flip)
    s.set_option(snch.OPT_PACKET, 0)
    b = s.query_silhouette(p, flip)
    assert torch.equal(a[0].view(torch.int32), b[0].view(torch.int32))
    assert (a[1] == b[1]).float().mean().item() > 0.999
    assert s.device_status() == 0
