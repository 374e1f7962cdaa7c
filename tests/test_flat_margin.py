"""The bound under which the 2D near-first searches take a leaf's box for no farther than
the leaf (scene2d.cu settled2), in float32 on the CPU: the mindist of the inflated box, as
computed, against the square of the distance, as computed, over random segments and points
of every scale that the bound admits, up to its edge."""
import numpy as np
import pytest

F = np.float32
LIMIT, NEAREST, SILHOUETTE, DISTANCE = F(16000), F(9), F(2), F(6)


def rounded(x):
    return np.asarray(x, np.float64).astype(F)


def mindist(a, b, p):
    off = F(1e-3)
    hi, lo = np.maximum(a, b) + off, np.minimum(a, b) - off
    d = np.minimum(hi, np.maximum(lo, p)) - p
    return d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]


def dot(u, v):
    return u[:, 0] * v[:, 0] + u[:, 1] * v[:, 1]


def segment_sq(a, b, p):
    u, v = b - a, p - a
    c1, c2 = dot(u, v), dot(u, u)
    with np.errstate(invalid="ignore", divide="ignore"):
        t = (c1 / c2)[:, None]
        w = p - (a + u * t)
    sq = dot(w, w)
    e = p - b
    sq = np.where(c2 <= c1, dot(e, e), sq)
    return np.where(c1 <= 0, dot(v, v), sq)


def cases(rng, n):
    """Segments of every length, at coordinates up to `m`, and points from on them to far off:
    half of them straight out from a box side or corner, where the margin is thinnest."""
    m = 10 ** rng.uniform(-2, 5.5, n)
    a = (rng.uniform(-1, 1, (n, 2))) * m[:, None]
    length = m * 10 ** rng.uniform(-7, 0.3, n)
    ang = rng.uniform(0, 2 * np.pi, n)
    ang = np.where(rng.random(n) < 0.3, np.round(ang / (np.pi / 2)) * (np.pi / 2), ang)
    b = a + (length[:, None] * np.stack([np.cos(ang), np.sin(ang)], 1))
    a, b = rounded(a), rounded(b)
    t = np.where(rng.random(n) < 0.5, np.round(rng.random(n)), rng.random(n))[:, None]
    on = a.astype(np.float64) * (1 - t) + b.astype(np.float64) * t
    far = m * 10 ** rng.uniform(-6, 0.8, n)
    dirn = rng.uniform(0, 2 * np.pi, n)
    dirn = np.where(rng.random(n) < 0.5, np.round(dirn / (np.pi / 4)) * (np.pi / 4), dirn)
    p = rounded(on + far[:, None] * np.stack([np.cos(dirn), np.sin(dirn)], 1))
    return a, b, p


@pytest.mark.parametrize("seed", range(4))
def test_boxes_stay_nearer_inside_the_bound(seed):
    rng = np.random.default_rng(seed)
    a, b, p = cases(rng, 1_000_000)
    top = np.abs(np.concatenate([a, b, p], 1)).max(1) + F(1e-3)
    md = mindist(a, b, p)
    sq = segment_sq(a, b, p)
    d = np.sqrt(sq)
    inside = NEAREST * top + DISTANCE * d <= LIMIT
    assert 0.3 < inside.mean() < 0.95
    assert np.all(md[inside] <= (d * d)[inside])
    # a vertex of the segment
    e = p - a
    dv = np.sqrt(dot(e, e))
    inside_v = SILHOUETTE * top + DISTANCE * dv <= LIMIT
    assert inside_v.mean() > inside.mean()
    assert np.all(md[inside_v] <= (dv * dv)[inside_v])
    # and the bound is there for a reason: far beyond it a box is farther than its segment
    far = np.float64(NEAREST) * top + DISTANCE * d > 40 * LIMIT
    if far.any():
        assert (md[far] > (d * d)[far]).any()


@pytest.mark.parametrize("seed", range(4))
def test_reach_at_every_scale(seed):
    """What lies beyond reach2 of a distance cannot hold an element at that distance, at any
    coordinates; and a box that contains another is never farther."""
    rng = np.random.default_rng(100 + seed)
    a, b, p = cases(rng, 1_000_000)
    big = rounded(10 ** rng.uniform(0, 4, len(a)))[:, None]
    a, b, p = a * big, b * big, p * big
    top = np.abs(np.concatenate([a, b, p], 1)).max(1) + F(1e-3)
    md = mindist(a, b, p)

    def reach(d, per_unit):
        r = d + (per_unit * top + DISTANCE * d) * F(2.0**-24)
        return r * r * F(1.0000019073486328125)

    d = np.sqrt(segment_sq(a, b, p))
    assert np.all(md <= reach(np.sqrt(d * d), NEAREST))
    e = p - a
    dv = np.sqrt(dot(e, e))
    assert np.all(md <= reach(dv, SILHOUETTE))
    c = rounded(a + rng.standard_normal(a.shape) * 10 ** rng.uniform(-4, 4, (len(a), 1)))
    lo, hi = np.minimum(np.minimum(a, b), c), np.maximum(np.maximum(a, b), c)
    assert np.all(mindist(lo, hi, p) <= md)
