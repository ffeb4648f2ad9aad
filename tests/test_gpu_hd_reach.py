"""The rule by which slivers count in the Hausdorff distance to a target of
256 triangles and more, restated on the CPU: the triangles in order, 32 at a
time, each with the lower bound (sqrt(q - e) - r)^2 and the upper bound q + e
of its centroid's squared distance q, as a bfloat16 contraction forms q; one
whose lower bound is above the smallest distance before its 32 and above the
smallest upper bound so far does not count. One sample stands at the centre of
a sphere of ordinary triangles that source and target share, so the distance
is that sample's; needles between the two, some of them with a float32
distance below their geometry's, are measured one at a time by the search that
counts every triangle. Tolerances: the distance itself is the same function's
(1e-5 relative), and cases in which a bound lies within 2e-6 of deciding
otherwise are left out."""
import importlib

import numpy as np
import pytest

from conftest import pkg

M, G = pkg("mesh"), pkg("meshgen")
T = importlib.import_module("cuacd-web_gb300.tree")

pytestmark = pytest.mark.gpu
R = 0.5
f32, f64 = np.float32, np.float64


def bf16_two(x):
    """x to two bfloat16 terms, each rounded to nearest even"""
    def one(v):
        b = v.astype(f32).view(np.uint32).astype(np.uint64)
        return ((b + 0x7FFF + ((b >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(f32)
    x = np.atleast_1d(np.asarray(x, f32))
    hi = one(x)
    return (hi + one(x - hi)).astype(f64)


def direct_sq(p, tri):
    """squared distance of p to a triangle, float64"""
    a, b, c = tri.astype(f64)
    n = np.cross(b - a, c - a)
    if n @ n > 0 and all(np.cross(v - u, p - u) @ n >= 0 for u, v in ((a, b), (b, c), (c, a))):
        return ((p - a) @ n) ** 2 / (n @ n)

    def seg(u, v):
        w = v - u
        s = np.clip((p - u) @ w / max(w @ w, 1e-300), 0, 1)
        return ((p - u - s * w) ** 2).sum()
    return min(seg(a, b), seg(b, c), seg(c, a))


def bounds(p, tris, split):
    """(lb, ub, slack) per triangle by the rule's formulas"""
    p = p.astype(f64)
    c = (tris.sum(1, dtype=f32) / f32(3)).astype(f64)
    r = np.sqrt(((tris.astype(f64) - c[:, None]) ** 2).sum(2)).max(1) * 1.00001 + 1e-30
    c2, p2 = (c * c).sum(1), p @ p
    if split:
        q = p2 + (bf16_two(-2 * c.ravel()).reshape(-1, 3) @ bf16_two(p) + bf16_two(c2))
    else:
        q = ((p - c) ** 2).sum(1)
    e = 2.0 ** -13 * (p2 + c2 + 2 * np.abs(p).sum() * np.abs(c).sum(1))
    lo = np.sqrt(np.maximum(q - e, 0)) - r
    return np.where(lo > 0, lo * lo, 0.0), q + e, 1e-10 * (p2 + c2) + 1e-30


def rule(b, v, nudge=0.0):
    """smallest distance of the triangles that count; nudge moves every lower
    bound by that share of the upper one"""
    lb, ub, slack = b
    best = run = 3.4e38
    for g in range(0, len(v), 32):
        s = slice(g, g + 32)
        up = np.minimum.accumulate(np.minimum(ub[s], run))
        keep = lb[s] + nudge * ub[s] <= np.minimum(best, up) * 1.001 + slack[s]
        run = up[-1]
        if keep.any():
            best = min(best, v[s][keep].min())
    return best


def scene(seed):
    """(p, ordinary triangles, needles): soups of corners (n, 3, 3)"""
    rng = np.random.default_rng([seed, 5])
    p = rng.uniform(-2.0, 2.0, 3).astype(f32)
    ico = G.icosphere(2)
    d = ico.verts.astype(f64)
    d *= R * rng.uniform(1.0, 1.02, (len(d), 1)) / np.linalg.norm(d, axis=1, keepdims=True)
    shell = (p + d).astype(f32)[ico.tris]

    def unit(n):
        u = rng.normal(size=(n, 3))
        return u / np.linalg.norm(u, axis=1, keepdims=True)
    m = 8  # ordinary triangles inside, the nearest among them
    mid = unit(m) * R * rng.uniform(0.86, 0.99, (m, 1))
    inner = (p + mid[:, None] + 0.02 * R * unit(3 * m).reshape(m, 3, 3)).astype(f32)
    inner = inner[~is_sliver(inner)]
    # needles: a, b, and a point of the line between, all but collinear
    k = 4088
    mid = unit(k) * R * rng.uniform(0.62, 0.93, (k, 1))
    u, h = unit(k), R * rng.uniform(0.02, 0.15, (k, 1))
    a, b = mid - h * u, mid + h * u
    out = np.maximum(np.linalg.norm(a, axis=1), np.linalg.norm(b, axis=1)) > 0.97 * R
    a[out], b[out] = mid[out] - 0.02 * R * u[out], mid[out] + 0.02 * R * u[out]
    w = unit(k) * 10.0 ** rng.uniform(-9.5, -8, (k, 1))
    needles = np.stack([a, b, a + rng.uniform(0.2, 0.8, (k, 1)) * (b - a) + w], 1)
    # a few exact segments whose middle is nearer to the centre than either
    # end: upper bounds far below their corners' distances
    q = np.zeros((8, 3, 3))
    axis = rng.integers(3, size=8)
    for i in range(8):
        q[i] = unit(1) * R * rng.uniform(0.4, 0.75)
        q[i, :, axis[i]] = np.array([-1, 1, rng.uniform(-0.2, 0.2)]) * R * 0.6
    return p, np.concatenate([shell, inner]), (p + np.concatenate([needles, q])).astype(f32), len(shell), rng


def soup(t):
    return M.Mesh(t.reshape(-1, 3).copy(), np.arange(3 * len(t), dtype=np.uint32).reshape(-1, 3))


def is_sliver(t):
    ab, ac = (t[:, 1] - t[:, 0]).astype(f64), (t[:, 2] - t[:, 0]).astype(f64)
    n2 = (np.cross(ab, ac) ** 2).sum(1)
    return n2 <= 1e-4 * (ab * ab).sum(1) * (ac * ac).sum(1)


def picks(needles, alone, p, rng):
    """a few needles whose measured distance is below their reach, up to 20
    others and now and then an exact segment (the last eight)"""
    lb = bounds(p, needles, True)[0]
    k = len(needles) - 8
    odd = np.flatnonzero(alone[:k] < 0.97 * np.minimum(lb[:k], alone.max()))
    rest = np.flatnonzero(alone[:k] >= lb[:k])
    n = int(rng.integers(1, 4)), int(rng.integers(0, 21)), int(rng.integers(0, 3))
    return np.concatenate([rng.permutation(odd)[: n[0]], rng.permutation(rest)[: n[1]],
                           k + rng.permutation(8)[: n[2]]])


# the needles' own samples lie nearer than this to the sphere or the centre: a
# smaller distance is not seen
FLOOR = 0.58 * R


class Scenes:
    def __init__(self):
        cfg = dict(width=3, width2=3, depth=1, nConcaveEdges=0, hullMaxVerts=4096, scratchWords=256 << 20)
        every, self.tree = T.GpuTree(**cfg, hdScreenMinTris=-1), T.GpuTree(**cfg)
        self.all = []
        for seed in range(6):
            p, plain, needles, ns, rng = scene(seed)
            assert is_sliver(needles).all() and not is_sliver(plain).any()
            # the source: the sphere and, at even places, triangles that are the point p
            src = soup(np.concatenate([np.broadcast_to(p, (4, 3, 3)), plain[:ns]]).astype(f32))
            alone = np.concatenate([
                every.hausdorff([(src, soup(np.concatenate([plain, t[None]]))) for t in needles[i:i + 1024]])
                for i in range(0, len(needles), 1024)]).astype(f64) ** 2
            base = np.array([direct_sq(p.astype(f64), t) for t in plain])
            self.all.append((seed, p, plain, needles, ns, rng, src, alone, base))

    def check(self, p, src, cases):
        """distances of the cases (triangles, their squared distances) against
        the rule; yields (want, bounds, squared distances, slivers)"""
        dist = self.tree.hausdorff([(src, soup(c[0])) for c in cases])
        for (tri, val), got in zip(cases, dist.astype(f64)):
            b = bounds(p, tri, True)
            want = rule(b, val)
            if any(rule(b, val, x) != want for x in (-2e-6, 2e-6)):
                continue
            if want < FLOOR ** 2:
                assert got <= FLOOR, (got, np.sqrt(want))
            else:
                assert abs(got - np.sqrt(want)) <= 1e-5 * got, (got, np.sqrt(want), np.sqrt(val.min()))
            yield want, b, val, is_sliver(tri)


@pytest.fixture(scope="module")
def scenes():
    return Scenes()


def differs(a, b):
    return max(a, FLOOR ** 2) != max(b, FLOOR ** 2)


def test_sliver_reach_rule(scenes):
    seen = dict(out=0, counts=0, odd=0, late=0)
    for seed, p, plain, needles, ns, rng, src, alone, base in scenes.all:
        cases = []
        for _ in range(512):
            some = picks(needles, alone, p, rng)
            o = rng.permutation(len(plain) + len(some))
            cases.append((np.concatenate([plain, needles[some]])[o], np.concatenate([base, alone[some]])[o]))
        for want, b, val, sliver in scenes.check(p, src, cases):
            first = np.concatenate([np.flatnonzero(~sliver), np.flatnonzero(sliver)])
            seen["out"] += differs(want, val.min())  # a sliver that does not count would decide
            seen["counts"] += differs(want, val[~sliver].min())  # one that counts does
            # ... below its reach, so that what comes before it decides
            seen["odd"] += differs(want, np.where(val < b[0], np.inf, val).min())
            seen["late"] += differs(want, rule(tuple(x[first] for x in b), val[first]))
    assert min(seen.values()) >= 3, seen


def radial(p, at, to=None):
    """an exact segment along the first axis through p, or across it at a
    distance: its normal is exactly zero, so it counts by its corners"""
    if to is None:
        t = np.array([[-0.64, at, 0], [0.64, at, 0], [0.1, at, 0]])
    else:
        t = np.array([[at, 0, 0], [to, 0, 0], [to - 0.01, 0, 0]])
    return (p + R * t).astype(f32)


def test_slivers_that_count_bound_what_follows(scenes):
    """A sliver that counts but is not the nearest triangle still rules out
    what is beyond it; a sliver whose centroid is near rules out ordinary
    triangles although it is far itself."""
    n = 0
    for seed, p, plain, needles, ns, rng, src, alone, base in scenes.all:
        shell, lb = plain[:ns], bounds(p, needles, True)[0]

        def near_at(x):
            d = rng.normal(size=3)
            d[0] = 0.0
            t = (p + x * d / np.linalg.norm(d) + 0.002 * R * rng.normal(size=(3, 3))).astype(f32)
            return t, direct_sq(p.astype(f64), t)
        cases = []
        for i in np.flatnonzero((alone < 0.9 * np.minimum(lb, base.min())) & (lb > 1.15 * FLOOR ** 2)).tolist()[:16]:
            # the nearest triangle last, beyond it the spoke's end, then the needle's reach
            spoke = radial(p, 0.985 * np.sqrt(lb[i]) / R, 0.97)
            v1, ub1 = direct_sq(p.astype(f64), spoke), bounds(p, spoke[None], True)[1][0]
            near, near2 = near_at(0.96 * np.sqrt(lb[i]))
            if is_sliver(near[None])[0] or not alone[i] < 0.95 * near2 < 0.95 * v1 or not lb[i] < 0.99 * ub1:
                continue
            for at in rng.integers(64, 288, size=4).tolist():
                tri = np.concatenate([shell[:10], spoke[None], shell[10:at], needles[i][None], shell[at:], near[None]])
                cases.append((tri, np.concatenate([base[:10], [v1], base[10:at], [alone[i]], base[at:ns], [near2]]), near2))
        n += len(cases)
        for case, (want, b, val, sliver) in zip(cases, scenes.check(p, src, [c[:2] for c in cases])):
            assert want == case[2]
        near, near2 = near_at(0.65 * R)
        bar = radial(p, 0.3)
        at = int(rng.integers(0, 300))
        tri = np.concatenate([shell[:at], bar[None], shell[at:], near[None]])
        corner = ((bar.astype(f64) - p.astype(f64)) ** 2).sum(1).min()
        val = np.concatenate([base[:at], [corner], base[at:ns], [near2]])
        got = list(scenes.check(p, src, [(tri, val)]))
        assert len(got) == 1 and got[0][0] == corner
    assert n >= 3


def tie(p, shell, needle, lb, width, rng):
    """the sphere with the needle and, right before it in its 32 triangles, an
    ordinary triangle whose upper bound is the needle's lower bound to a share
    of `width`"""
    d = rng.normal(size=3)
    d /= np.linalg.norm(d)
    shape = 0.01 * R * rng.normal(size=(3, 3))
    lo, hi, goal = 0.0, 1.2 * R, lb * (1 + rng.uniform(-width, width)) / 1.001
    for _ in range(60):
        mid = (lo + hi) / 2
        t = (p + mid * d + shape).astype(f32)
        if bounds(p, t[None], False)[1][0] < goal:
            lo = mid
        else:
            hi = mid
    at = 2 * int(rng.integers(1, len(shell) // 2))
    return np.concatenate([shell[:at], t[None], needle[None], shell[at:]]), at


def test_reach_uses_split_coordinates(scenes):
    """Where the two forms of |p - c|^2 decide differently, the split one does."""
    n = 0
    for seed, p, plain, needles, ns, rng, src, alone, base in scenes.all:
        (lb, ub, _), other = bounds(p, needles, True), bounds(p, needles, False)
        width = 2 * np.median(np.abs(lb - other[0]) / ub)
        cases = []
        for i in np.flatnonzero((alone < 0.9 * np.minimum(lb, base.min())) & (lb < 0.95 * R * R)
                                & (lb > FLOOR ** 2)).tolist()[:16]:
            for _ in range(24):
                tri, at = tie(p, plain[:ns], needles[i], lb[i], width, rng)
                val = np.insert(base[:ns], at, [direct_sq(p.astype(f64), tri[at]), alone[i]])
                if not is_sliver(tri[at:at + 1])[0] and \
                        differs(rule(bounds(p, tri, True), val), rule(bounds(p, tri, False), val)):
                    cases.append((tri, val))
        n += sum(1 for _ in scenes.check(p, src, cases)) if cases else 0
    assert n >= 3, n
