"""The work a user of the engine has it do, as cases that can be timed.

Every case goes through the public Python entry points (GpuTree, Decomposer)
as a program calls them: host meshes in, host results out. A program keeps
one tree or decomposer per configuration and feeds it new meshes, so handles
are kept per configuration here too; what `prepare` makes anew from the seed
is the input meshes, planes and pairs.

Kinds
  hulls     GpuTree.hull_meshes: exact convex hulls with their faces
  hausdorff GpuTree.hausdorff: sampled Hausdorff distance of mesh pairs
  hullshd   GpuTree.hulls_with_hausdorff: new halves' hulls and distances
  cuts      GpuTree.plane_cuts: capped plane cuts, both halves read back
  concave   GpuTree.concave_planes: candidate planes from concave edges
  tree      GpuTree.run: the lookahead tree with refinement rounds
  eval      GpuTree.eval_cuts: cut, hulls, rv and Hausdorff per candidate
  decompose Decomposer.decompose: the whole loop with its merge pass
"""
from __future__ import annotations

import importlib
import json
import math

import numpy as np
import torch

_PKG = "cuacd-web_gb300."


def _mod(name):
    return importlib.import_module(_PKG + name)


# ---------------------------------------------------------------------------
# the cases


def listed():
    return [
        # one tree child: the smallest call a program makes (latency)
        dict(name="hull_one_part", kind="hulls", shape="points", n=1, lo=150, hi=150),
        # a merge round's pair hulls: unions of two parts' hull vertices
        dict(name="hulls_merge_pairs", kind="hulls", shape="points", n=512, lo=40, hi=1000),
        # the first hull of a large organic mesh (56k triangles)
        dict(name="hull_large_mesh", kind="hulls", shape="blob", n=1, lo=56000, hi=56000),
        # the merge pass's distances: parts against their hulls
        dict(name="hausdorff_pairs", kind="hausdorff", n=192, lo=160, hi=6000),
        # an iteration's new halves in one batch: hulls and distances
        dict(name="hulls_hd_halves", kind="hullshd", n=24, lo=1500, hi=30000),
        # 96 candidate planes of a 5,120-triangle noisy icosphere, cut at once
        dict(name="cuts_icosphere", kind="cuts", shape="icosphere", n=96, lo=5120, hi=5120),
        # the winning cuts of a batch of meshes: one plane each, closed parts
        dict(name="cuts_batch", kind="cuts", shape="blob", n=12, lo=1000, hi=56000),
        # concave-edge planes of an uneven batch
        dict(name="concave_batch", kind="concave", n=16, lo=500, hi=56000, edges=16),
        # the lookahead tree on 160 small parts at depth 3 with two refinement rounds
        dict(name="tree_staircases", kind="tree", shape="staircase", n=160, lo=188, hi=188, width=6, depth=3),
        # the lookahead tree on a few large parts at depth 2
        dict(name="tree_blobs", kind="tree", shape="blob", n=3, lo=3000, hi=24000, width=6, depth=2),
        # cut, hull, rv and Hausdorff of both halves of 96 candidate planes
        dict(name="eval_icosphere", kind="eval", shape="icosphere", n=96, lo=5120, hi=5120),
        # a mesh decomposed from start to end, merge pass included
        dict(name="decompose_blob", kind="decompose", n=1, lo=8000, hi=8000, threshold=0.05, iters=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the listed ones' kinds, its sizes between the smallest
    and the largest a program meets there."""
    k = rng.choice(["hulls", "hulls", "hausdorff", "hullshd", "cuts", "cuts", "concave", "tree", "eval", "decompose"])
    if k == "hulls":
        if rng.random() < 0.5:
            hi = _log(rng, 100, 1000)
            return dict(kind=k, shape="points", n=_log(rng, 1, 512), lo=_log(rng, 40, hi), hi=hi)
        hi = _log(rng, 2500, 56000)
        return dict(kind=k, shape="blob", n=1 if hi > 20000 else rng.randint(1, 4), lo=_log(rng, 2000, hi), hi=hi)
    if k == "hausdorff":
        hi = _log(rng, 300, 6000)
        return dict(kind=k, n=_log(rng, 1, 192), lo=_log(rng, 150, hi), hi=hi)
    if k == "hullshd":
        hi = _log(rng, 2000, 30000)
        return dict(kind=k, n=2 * rng.randint(1, 12), lo=_log(rng, 1500, hi), hi=hi)
    if k == "cuts":
        if rng.random() < 0.5:
            level = rng.choice([2, 3, 4])
            return dict(kind=k, shape="icosphere", n=_log(rng, 1, 96), lo=20 * 4 ** level, hi=20 * 4 ** level)
        hi = _log(rng, 1500, 56000)
        return dict(kind=k, shape="blob", n=rng.randint(1, 12), lo=_log(rng, 1000, hi), hi=hi)
    if k == "concave":
        hi = _log(rng, 600, 56000)
        return dict(kind=k, n=rng.randint(1, 16), lo=_log(rng, 500, hi), hi=hi, edges=rng.choice([8, 16, 32]))
    if k == "tree":
        if rng.random() < 0.5:
            steps = rng.randint(4, 8)
            nt = 188 * steps // 8
            return dict(kind=k, shape="staircase", n=_log(rng, 1, 160), lo=nt, hi=nt, width=rng.choice([3, 6]),
                        depth=rng.choice([2, 3]))
        hi = _log(rng, 2000, 24000)
        return dict(kind=k, shape="blob", n=rng.randint(1, 3), lo=_log(rng, 1500, hi), hi=hi, width=6, depth=2)
    if k == "eval":
        return dict(kind=k, shape="icosphere", n=_log(rng, 4, 96), lo=5120, hi=5120)
    size = _log(rng, 1200, 5000)
    return dict(kind=k, n=1, lo=size, hi=size, threshold=rng.choice([0.05, 0.1]), iters=rng.randint(3, 7))


# ---------------------------------------------------------------------------
# inputs


def _sizes(case, rng):
    """The case's n sizes, log-evenly spread from lo to hi, in seeded order."""
    n, lo, hi = case["n"], case["lo"], case["hi"]
    s = np.exp(np.log(lo) + (np.arange(n) + 0.5) / n * (np.log(hi) - np.log(lo)))
    return [int(x) for x in rng.permutation(np.round(s))]


def _blob(tris, rng):
    """A blob isosurface of about `tris` triangles, extent 2."""
    gen = _mod("meshgen")
    nb, seed = int(rng.integers(6, 25)), int(rng.integers(1 << 30))
    m0 = gen.blob_mesh(nb, 24, seed=seed)
    g = int(np.clip(round(24 * np.sqrt(tris / max(m0.nt, 1))), 8, 120))
    return _mod("mesh").normalize(m0 if g == 24 else gen.blob_mesh(nb, g, seed=seed))[0]


def _pair_union(n, rng):
    """About n points: the vertices of two neighbouring rounded hulls."""
    out = []
    for k, c in ((0, n // 2), (1, n - n // 2)):
        p = rng.normal(size=(c, 3))
        p /= np.linalg.norm(p, axis=1, keepdims=True)
        p *= rng.uniform(0.3, 0.6, size=3) * rng.uniform(0.97, 1.0, size=(c, 1))
        p[:, 0] += (0.45, -0.45)[k]
        out.append(p)
    Mesh = _mod("mesh").Mesh
    return Mesh(np.concatenate(out).astype(np.float32), np.zeros((0, 3), np.uint32))


def _icosphere(tris, rng):
    level = int(round(math.log(tris / 20, 4)))
    return _mod("meshgen").noisy_icosphere(level, seed=int(rng.integers(1 << 30)))


def _mid_plane(m, rng):
    """A plane through the middle half of the mesh, as winning cuts are."""
    n = rng.normal(size=3)
    n /= np.linalg.norm(n)
    p = m.verts.astype(np.float64) @ n
    return [*n, -(p.min() + rng.uniform(0.25, 0.75) * (p.max() - p.min()))]


def _inputs(case, seed):
    rng = np.random.default_rng([seed, 77])
    k = case["kind"]
    if k == "hulls":
        make = _pair_union if case["shape"] == "points" else _blob
        return dict(meshes=[make(s, rng) for s in _sizes(case, rng)])
    if k == "hausdorff":
        # parts of a few meshes at several resolutions against their hulls
        Mesh = _mod("mesh").Mesh
        parts = [_blob(s, rng) for s in _sizes(dict(case, n=min(case["n"], 24)), rng)]
        g = _tree(hullMaxVerts=16384)
        hulls, _ = g.hull_meshes(parts)
        base = [(p, Mesh(p.verts, h["tris"])) for p, h in zip(parts, hulls)]
        pairs = []
        for i in range(case["n"]):
            a, b = base[i % len(base)]
            s = rng.uniform(0.25, 1.0, size=3).astype(np.float32)  # parts differ in extent
            pairs.append((Mesh(a.verts * s, a.tris), Mesh(b.verts * s, b.tris)))
        return dict(pairs=pairs)
    if k == "hullshd":
        cut = _mod("decompose").plane_cut
        halves = []
        for s in _sizes(dict(case, n=case["n"] // 2), rng):
            m = _blob(2 * s, rng)
            halves += cut(m, _mid_plane(m, rng))
        return dict(meshes=halves)
    if k in ("cuts", "eval"):
        if case["shape"] == "icosphere":
            m = _icosphere(case["lo"], rng)
            planes = _mod("meshgen").random_planes(m, case["n"], seed=int(rng.integers(1 << 30)))
            return dict(meshes=[m], planes=planes, of=[0] * case["n"])
        meshes = [_blob(s, rng) for s in _sizes(case, rng)]
        return dict(meshes=meshes, planes=[_mid_plane(m, rng) for m in meshes], of=list(range(case["n"])))
    if k == "concave":
        return dict(meshes=[_blob(s, rng) for s in _sizes(case, rng)],
                    seeds=[int(x) for x in rng.integers(1 << 31, size=case["n"])])
    if k == "tree":
        conc, Mesh = _mod("concave"), _mod("mesh").Mesh
        if case["shape"] == "staircase":
            base = _mod("mesh").normalize(_mod("meshgen").staircase(max(1, round(case["lo"] / 23.5)), wall_centroids=True))[0]
            meshes = [Mesh(base.verts * rng.uniform(0.6, 1.0, size=3).astype(np.float32), base.tris)
                      for _ in range(case["n"])]
        else:
            meshes = [_blob(s, rng) for s in _sizes(case, rng)]
        planes = [conc.concave_edge_planes(m, 16) for m in meshes]
        spacing = conc.refine_spacing(meshes, 0.1, case["width"])
        return dict(meshes=meshes, planes=planes, refine=dict(rounds=2, probes=8, spacing=spacing))
    return dict(meshes=[_blob(s, rng) for s in _sizes(case, rng)])


# ---------------------------------------------------------------------------
# handles: one per configuration, as a program keeps them

_handles = {}
_POOLS = dict(vertexCap=96 << 20, triCap=96 << 20, edgeCap=8 << 20, scratchWords=96 << 20, hullBudgetBytes=6 << 30)


def _tree(**cfg):
    cfg = dict(dict(width=3, width2=3, depth=1, nConcaveEdges=0, hullMaxVerts=32768), **_POOLS, **{**cfg})
    key = "tree" + json.dumps(cfg, sort_keys=True)
    if key not in _handles:
        _handles[key] = _mod("tree").GpuTree(**cfg)
    return _handles[key]


def _decomposer(**opts):
    key = "dec" + json.dumps(opts, sort_keys=True)
    if key not in _handles:
        _handles[key] = _mod("decompose").Decomposer(**opts, tree=dict(_POOLS, hullMaxVerts=32768))
    return _handles[key]


def prepare(case, seed):
    s = _inputs(case, seed)
    k = case["kind"]
    if k == "tree":
        s["handle"] = _tree(width=case["width"], width2=3, depth=case["depth"], nConcaveEdges=16, minEdgeDist=0.015,
                            hullMaxVerts=16384)
    elif k == "decompose":
        s["handle"] = _decomposer(threshold=case["threshold"], width=6, width2=3, depth=2, maxIters=case["iters"])
    else:
        s["handle"] = _tree()
    s["case"] = case
    return s


# ---------------------------------------------------------------------------
# one pass


def _rows(arrays, dtype, width, rows):
    """The arrays one after another in a buffer of `rows` rows, zeros behind."""
    n = sum(len(a) for a in arrays)
    out = np.zeros((max(rows, n), width), dtype)
    at = 0
    for a in arrays:
        out[at:at + len(a)] = a
        at += len(a)
    return out


def _room(case):
    """Rows for a case's triangles: results' sizes follow the data, buffers
    that a program keeps them in do not."""
    t = _total(case)
    if case["kind"] == "cuts":
        each = case["lo"] if case["shape"] == "icosphere" else t / case["n"]
        return int(case["n"] * (1.5 * each + 40 * math.sqrt(each)))
    if case["kind"] == "decompose":
        return int(8 * t)
    return int(2 * t)


def run(s):
    c, g = s["case"], s["handle"]
    k = c["kind"]
    if k == "hulls":
        hulls, status = g.hull_meshes(s["meshes"])
        return dict(status=status, tris=_rows([h["tris"] for h in hulls if h], np.uint32, 3, _room(c)),
                    volume=np.array([h["volume"] if h else 0.0 for h in hulls], np.float32))
    if k == "hausdorff":
        return dict(distance=g.hausdorff(s["pairs"]))
    if k == "hullshd":
        hulls = g.hulls_with_hausdorff(s["meshes"])
        return dict(status=np.array(g.last_hull_fails),
                    tris=_rows([h["tris"] for h in hulls if h], np.uint32, 3, _room(c)),
                    volume=np.array([h["volume"] if h else 0.0 for h in hulls], np.float32),
                    distance=np.array([h["hausdorff"] if h else 0.0 for h in hulls], np.float32))
    if k == "cuts":
        r = g.plane_cuts(s["meshes"], s["planes"], s["of"], closed=True)
        halves = [h for x in r if x[0] == 0 for h in x[1:]]
        return dict(status=np.array([x[0] for x in r]),
                    nv=np.array([[h.nv if h else 0 for h in x[1:]] for x in r]),
                    verts=_rows([h.verts for h in halves], np.float32, 3, _room(c)),
                    tris=_rows([h.tris for h in halves], np.uint32, 3, _room(c)))
    if k == "concave":
        p = g.concave_planes(s["meshes"], c["edges"], seeds=s["seeds"])
        return dict(count=np.array([len(x) for x in p]), planes=_rows(p, np.float32, 4, 4 * c["n"] * c["edges"]))
    if k == "tree":
        r = g.run(s["meshes"], s["planes"], refine=s["refine"])
        return dict(cut=np.array([x["bestCut"] for x in r["seeds"]]),
                    cost=np.array([x["bestCost"] for x in r["seeds"]], np.float32),
                    plane=np.array([x["plane"] or [0.0] * 4 for x in r["seeds"]], np.float32),
                    counts=np.array([r["validJobs"], r["pruned"], r["hullFailCount"], int(r["overflow"])]))
    if k == "eval":
        o = g.eval_cuts(s["meshes"][0], s["planes"])
        return dict(split=o[:, 0].astype(np.int64), volume=o[:, 1:3].copy(), hull=o[:, 3:5].copy(),
                    rv=o[:, 5:7].copy(), distance=o[:, 7].copy())
    r = g.decompose(s["meshes"][0])
    parts = r.parts
    return dict(iterations=r.iterations,
                sizes=_rows([[[p.mesh.nv, p.mesh.nt, p.hull.nv, p.hull.nt]] for p in parts], np.int64, 4, 256),
                verts=_rows([p.mesh.verts for p in parts], np.float32, 3, _room(c)),
                tris=_rows([p.mesh.tris for p in parts], np.uint32, 3, _room(c)),
                hull_verts=_rows([p.hull.verts for p in parts], np.float32, 3, _room(c)),
                hull_tris=_rows([p.hull.tris for p in parts], np.uint32, 3, _room(c)),
                volumes=_rows([[[p.meshVol, p.hullVol, p.hausdorff or 0.0]] for p in parts], np.float64, 3, 256))


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _total(case):
    """Sum of the case's sizes (triangles, or points of a point set)."""
    n = case["n"] // 2 if case["kind"] == "hullshd" else case["n"]
    lo, hi = case["lo"], case["hi"]
    s = sum(math.exp(math.log(lo) + (i + 0.5) / n * (math.log(hi) - math.log(lo))) for i in range(n))
    return 2.2 * s if case["kind"] == "hullshd" else s


def work(case):
    """Bytes: inputs read once (12 per vertex, 12 per triangle, half as many
    vertices as triangles) and outputs written once. Flops: one plane or
    distance evaluation per element where an algorithm must at least look at
    every element once, in units of the operation's own count."""
    k, t = case["kind"], _total(case)
    mesh = 18.0 * t
    if k == "hulls":
        pts = t if case["shape"] == "points" else t / 2
        faces = pts * (1.0 if case["shape"] == "points" else 0.2)
        return dict(bytes=12 * pts + 12 * faces, flops=16 * pts)
    if k == "hausdorff":
        # every sample of either side against its nearest triangle at least
        return dict(bytes=2.0 * 18 * t + 4 * case["n"], flops=2.0 * 2000 * case["n"] * 70)
    if k == "hullshd":
        return dict(bytes=mesh + 1.2 * t, flops=8.0 * t + 2.0 * 3000 * case["n"] * 70)
    if k == "cuts":
        cuts = case["n"] * case["lo"] if case["shape"] == "icosphere" else t
        read = 18.0 * case["lo"] if case["shape"] == "icosphere" else mesh
        return dict(bytes=read + 18.0 * cuts, flops=3.5 * cuts)
    if k == "concave":
        return dict(bytes=mesh + 64.0 * case["n"] * case["edges"], flops=60.0 * t)
    if k == "tree":
        # every job reads its parent once, writes its two children's points
        # and the hulls read them once, over the levels and two probe rounds
        cuts0 = 64 + case["width"] if case["shape"] == "staircase" else 40
        jobs = sum(cuts0 * 3 ** l for l in range(case["depth"])) + 2 * sum(8 * 3 ** l for l in range(case["depth"]))
        return dict(bytes=0.5 * jobs * 30.0 * t, flops=0.5 * jobs * 30.0 * t)
    if k == "eval":
        cuts = case["n"] * case["lo"]
        return dict(bytes=18.0 * case["lo"] + 36.0 * cuts, flops=20.0 * cuts + 2 * 2.0 * 2000 * case["n"] * 70)
    # the whole loop: a tree per iteration over parts that sum to the mesh
    return dict(bytes=case["iters"] * 30 * 15.0 * t, flops=case["iters"] * 30 * 30.0 * t)


# ---------------------------------------------------------------------------
# the same results in 64 bits


def _hull_volume(points):
    """Volume of the convex hull, float64: farthest-point insertion over
    faces kept as arrays, outside points reassigned to the new faces."""
    p = np.unique(points.astype(np.float64), axis=0)
    if len(p) < 4:
        return 0.0
    scale = float(np.ptp(p, axis=0).max())
    if scale <= 0:
        return 0.0
    p = (p - p.mean(0)) / scale
    eps = 1e-13
    i0 = int(p[:, 0].argmin())
    i1 = int(((p - p[i0]) ** 2).sum(1).argmax())
    d = np.cross(p[i1] - p[i0], p - p[i0])
    i2 = int((d ** 2).sum(1).argmax())
    n = np.cross(p[i1] - p[i0], p[i2] - p[i0])
    h = (p - p[i0]) @ n
    i3 = int(np.abs(h).argmax())
    if abs(h[i3]) < 1e-14:
        return 0.0
    if h[i3] > 0:
        i1, i2 = i2, i1
    F = [[i0, i1, i2], [i0, i3, i1], [i1, i3, i2], [i2, i3, i0]]

    def plane(f):
        f = np.asarray(f)
        q = np.cross(p[f[:, 1]] - p[f[:, 0]], p[f[:, 2]] - p[f[:, 0]])
        q /= np.maximum(np.linalg.norm(q, axis=1, keepdims=True), 1e-300)
        return q, (q * p[f[:, 0]]).sum(1)

    F = np.array(F)
    N, D = plane(F)
    owner = np.full(len(p), -1)
    dist = np.zeros(len(p))

    def assign(idx, f0):
        for a in range(0, len(idx), 4096):
            i = idx[a:a + 4096]
            v = p[i] @ N[f0:].T - D[f0:]
            b = v.argmax(1)
            m = v[np.arange(len(i)), b]
            out = m > eps
            owner[i] = np.where(out, b + f0, -1)
            dist[i] = np.where(out, m, 0.0)

    assign(np.arange(len(p)), 0)
    while True:
        k = int(dist.argmax())
        if dist[k] <= eps:
            break
        vis = N @ p[k] - D > eps
        vis[owner[k]] = True
        tri = F[vis]
        e = np.concatenate([tri[:, [0, 1]], tri[:, [1, 2]], tri[:, [2, 0]]])
        key, rev = e[:, 0] * len(p) + e[:, 1], e[:, 1] * len(p) + e[:, 0]
        rim = e[~np.isin(key, rev)]
        new = np.concatenate([rim, np.full((len(rim), 1), k)], 1)
        orphans = np.flatnonzero((owner >= 0) & vis[np.maximum(owner, 0)])
        renum = np.cumsum(~vis) - 1
        live = owner >= 0
        owner[live] = renum[owner[live]]
        f0 = int((~vis).sum())
        qn, qd = plane(new)
        F, N, D = np.concatenate([F[~vis], new]), np.concatenate([N[~vis], qn]), np.concatenate([D[~vis], qd])
        owner[k], dist[k] = -1, 0.0
        orphans = orphans[orphans != k]
        if len(orphans):
            assign(orphans, f0)
    return float(np.abs((p[F[:, 0]] * np.cross(p[F[:, 1]], p[F[:, 2]])).sum() / 6.0)) * scale ** 3


def _samples(m):
    """The distance's surface samples: counts by area share, at least one on
    every second (or step-th) triangle, barycentrics from a Wang hash."""
    a, b, c = (m.verts.astype(np.float64)[m.tris[:, q]] for q in range(3))
    area = 0.5 * np.linalg.norm(np.cross(b - a, c - a), axis=1)
    res = max(1000.0, math.floor(2000.0 * area.sum()))
    nt = len(area)
    cnt = np.floor(res / area.sum() * area).astype(np.int64)
    every = max(nt // int(res), 1) if nt > res else 2
    cnt = np.where(cnt > 0, cnt, (np.arange(nt) % every == 0).astype(np.int64))
    t = np.repeat(np.arange(nt), cnt)
    j = np.arange(len(t)) - np.repeat(np.cumsum(cnt) - cnt, cnt)

    def wang(s):
        s = (s ^ np.uint32(61)) ^ (s >> np.uint32(16))
        s = s * np.uint32(9)
        s = s ^ (s >> np.uint32(4))
        s = s * np.uint32(0x27D4EB2D)
        return s ^ (s >> np.uint32(15))

    ha = wang((t * 65537 + j).astype(np.uint64).astype(np.uint32))
    hb = wang(ha + np.uint32(0x9E3779B9))
    ra, rb = (h.astype(np.float64) % (1 << 24) / ((1 << 24) - 1) for h in (ha, hb))
    q = np.sqrt(ra)
    return (1 - q)[:, None] * a[t] + (q * (1 - rb))[:, None] * b[t] + (q * rb)[:, None] * c[t]


def _directed(samples, m, dev):
    """Largest distance of the samples to the mesh, float64, brute force."""
    p = torch.from_numpy(samples).to(dev)
    a, b, c = (torch.from_numpy(m.verts.astype(np.float64)[m.tris[:, q]]).to(dev) for q in range(3))
    worst = 0.0

    def seg(x, u, v):
        w = v - u
        s = ((x - u) * w).sum(-1) / (w * w).sum(-1).clamp_min(1e-300)
        return ((x - u - s.clamp(0, 1)[..., None] * w) ** 2).sum(-1)

    n = torch.linalg.cross(b - a, c - a)
    n2 = (n * n).sum(-1)
    for i in range(0, len(p), max(1, (1 << 21) // len(a))):
        x = p[i:i + max(1, (1 << 21) // len(a)), None, :]
        best = torch.minimum(torch.minimum(seg(x, a, b), seg(x, b, c)), seg(x, c, a))
        side = [(torch.linalg.cross((v - u).expand_as(x - u), x - u) * n).sum(-1) >= 0
                for u, v in ((a, b), (b, c), (c, a))]
        inside = side[0] & side[1] & side[2] & (n2 > 1e-20)
        flat = ((x - a) * n).sum(-1) ** 2 / n2.clamp_min(1e-300)
        best = torch.where(inside, torch.minimum(best, flat), best)
        worst = max(worst, float(best.min(-1).values.max()))
    return math.sqrt(worst)


def _half_surfaces(m, plane):
    """Both halves' surface triangles in input order with their vertices in
    first-use order, float64; None when the plane does not split the mesh."""
    pl = np.asarray(plane, np.float64)
    ln = float(np.linalg.norm(pl[:3]))
    n, d0 = pl[:3] / ln, pl[3] / ln
    v = m.verts.astype(np.float64)
    d = v @ n + d0
    s = np.where(d > 1e-6, 1, np.where(d < -1e-6, -1, 0))
    if not (s > 0).any() or not (s < 0).any():
        return None
    extra, ids, out = [], {}, []
    tris, st = m.tris.tolist(), s[m.tris].tolist()
    for keep in (1, -1):
        poly = []
        for (t, g) in zip(tris, st):
            if g[0] == g[1] == g[2] == 0:
                continue
            if keep * g[0] >= 0 and keep * g[1] >= 0 and keep * g[2] >= 0:
                poly.append(t)
                continue
            if keep * g[0] <= 0 and keep * g[1] <= 0 and keep * g[2] <= 0:
                continue
            q = []
            for k in range(3):
                i, j = t[k], t[(k + 1) % 3]
                if keep * g[k] >= 0:
                    q.append(i)
                if g[k] * g[(k + 1) % 3] < 0:
                    e = (min(i, j), max(i, j))
                    if e not in ids:
                        ids[e] = len(v) + len(extra)
                        x = d[e[0]] / (d[e[0]] - d[e[1]])
                        extra.append(v[e[0]] + x * (v[e[1]] - v[e[0]]))
                    q.append(ids[e])
            poly += [[q[0], q[k], q[k + 1]] for k in range(1, len(q) - 1)]
        out.append(np.array(poly, np.int64))
    every = np.concatenate([v, np.array(extra).reshape(-1, 3)])
    halves = []
    for f in out:
        u, first = np.unique(f.ravel(), return_index=True)
        halves.append((every[u[np.argsort(first)]], every[f]))
    return halves, n, d0


def _concave(m, edges, seed, eps=0.005, thr=3.49):
    """Face-offset and bisector planes of a seeded reservoir of the concave
    edges, float64."""
    v, t = m.verts.astype(np.float64), m.tris.astype(np.int64)
    src, dst = t.ravel(), t[:, [1, 2, 0]].ravel()
    face = np.repeat(np.arange(len(t)), 3)
    key = src * m.nv + dst
    order = np.argsort(key, kind="stable")
    uk, first = np.unique(key[order], return_index=True)
    low = face[order][first]
    a, b = uk // m.nv, uk % m.nv
    rev = np.searchsorted(uk, b * m.nv + a).clip(max=len(uk) - 1)
    sel = (a < b) & (uk[rev] == b * m.nv + a)
    f0, f1 = np.minimum(low, low[rev])[sel], np.maximum(low, low[rev])[sel]
    a, b = a[sel], b[sel]
    n = np.cross(v[t[:, 1]] - v[t[:, 0]], v[t[:, 2]] - v[t[:, 0]])
    ln = np.linalg.norm(n, axis=1)
    unit = n / np.maximum(ln, 1e-300)[:, None]
    n0, n1 = unit[f0], unit[f1]
    alpha = np.arccos(np.clip((n0 * n1).sum(1), -1, 1))
    tf = t[f0]
    other = np.where((tf != a[:, None]) & (tf != b[:, None]), tf, -1).max(1)
    side = ((v[other] - v[a]) * n1).sum(1)
    ok = (ln[f0] >= 1e-12) & (ln[f1] >= 1e-12) & (np.where(side > 0, math.pi + alpha, math.pi - alpha) > thr)
    kept, rng = [], seed & 0xFFFFFFFF
    for seen, i in enumerate(np.flatnonzero(ok).tolist(), 1):
        if len(kept) < edges:
            kept.append(i)
            continue
        rng = (rng * 1664525 + 1013904223) & 0xFFFFFFFF
        if rng < math.floor(edges / seen * 4294967295.0):
            rng = (rng * 1664525 + 1013904223) & 0xFFFFFFFF
            kept[rng % edges] = i
    out = []
    for i in kept:
        p = (v[a[i]] + v[b[i]]) / 2
        out += [[*q, -(q @ p + eps)] for q in (n1[i], n0[i])]
        q = n0[i] + n1[i]
        ql = np.linalg.norm(q)
        if ql >= 1e-4:
            q = q / ql
            out += [[*q, -(q @ p + eps)], [*q, -(q @ p - eps)]]
    return np.array(out).reshape(-1, 4)


def exact(case, seed):
    k = case["kind"]
    if k in ("tree", "decompose"):
        return None  # a search's result: its costs have no closed form
    s = _inputs(case, seed)
    if k == "hulls":
        return dict(status=None, tris=None, volume=np.array([_hull_volume(m.verts) for m in s["meshes"]]))
    if k == "hausdorff":
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        return dict(distance=np.array([max(_directed(_samples(a), b, dev), _directed(_samples(b), a, dev))
                                       for a, b in s["pairs"]]))
    if k == "hullshd":
        # the hull side's samples follow its face order: no value without it
        return dict(status=None, tris=None, distance=None,
                    volume=np.array([_hull_volume(m.verts) for m in s["meshes"]]))
    if k == "cuts":
        found = [_half_surfaces(s["meshes"][i], p) for i, p in zip(s["of"], s["planes"])]
        return dict(status=None, nv=None, tris=None,
                    verts=_rows([h[0] for f in found if f for h in f[0]], np.float64, 3, _room(case)))
    if k == "concave":
        return dict(count=None, planes=_rows([_concave(m, case["edges"], x) for m, x in zip(s["meshes"], s["seeds"])],
                                             np.float64, 4, 4 * case["n"] * case["edges"]))
    vol, hull, rv = (np.zeros((case["n"], 2)) for _ in range(3))
    for i, p in enumerate(s["planes"]):
        f = _half_surfaces(s["meshes"][0], p)
        for j, (verts, tri) in enumerate(f[0] if f else []):
            q = (tri.astype(np.float32).astype(np.float64) + f[1] * f[2]).transpose(1, 0, 2)  # the plane through 0
            vol[i, j] = abs((q[0] * np.cross(q[1], q[2])).sum() / 6)
            hull[i, j] = _hull_volume(verts.astype(np.float32))
            rv[i, j] = 0.3 * np.cbrt(3 / (4 * math.pi) * max(hull[i, j] - vol[i, j], 0.0))
    return dict(split=None, distance=None, volume=vol, hull=hull, rv=rv)
