"""Timed cases of the spatial join: what a program does with this package, through its public entry points.

A case is a dict of plain values.  Its "kind" names the call:

  join    a join of two tiles that are resident on the GPU (or of one with
          itself): kNN or within, FP32 result bounds or exact FP64 distances
  attach  the same from page-locked host bytes: both tiles attached, joined
          and released, every pass
  serve   a burst of requests to the request loop over a resident vessel tile
  refine  the batched voxel-pair refine on host arrays
  prep    LOD preparation: meshes in, a RAW tile with LODs, voxels and bounds out

The tiles are the package's synthetic workload (nuclei of 320 or 1280 triangles
around vessels of about 20k triangles, five LODs) in the shapes of its
benchmark and tests; every size below is a vessel count and a nuclei count per
vessel of that workload.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

tdp = importlib.import_module("3dpipe_b200").tdp

_JOIN = {"kind": "join", "query": "within", "knn": 0, "within": 0.0, "self": False, "exact": False, "autotune": False,
         "level": 2, "lods": "", "subdiv": 3, "voxel_size": 100}


def _case(name, **kw):
    kind = kw.get("kind", "join")
    base = dict(_JOIN) if kind in ("join", "attach") else {}
    base.update(kw)
    return {"name": name, **base} if name else base


def listed():
    return [
        # the smallest join of the benchmark's configurations: an interactive
        # query, all launches and round trips
        _case("nn10_small", query="nn", knn=10, vessels=10, per_vessel=20),
        # an ordinary analysis on one field of view, as `tdbase join` runs it
        _case("within150_ordinary", within=150.0, vessels=100, per_vessel=20),
        # the headline join (within 400), a tenth of the benchmark's tile, on a
        # context that the program autotuned once
        _case("within400_large", within=400.0, vessels=100, per_vessel=200, autotune=True),
        # nearest vessels of every nucleus of a large tile
        _case("nn10_large", query="nn", knn=10, vessels=100, per_vessel=200),
        # nearest neighbours among the nuclei themselves: many candidates,
        # refine-bound
        _case("nn10_self", query="nn", knn=10, vessels=20, per_vessel=150, self=True, autotune=True),
        # neighbours within a cell-to-cell distance, ragged sizes, smaller voxels
        _case("within60_self_odd", within=60.0, vessels=37, per_vessel=113, self=True, voxel_size=70),
        # exact FP64 distances of every reported pair
        _case("exact_within150", within=150.0, vessels=50, per_vessel=20, exact=True),
        # tiles streamed from host memory: nothing resident before the call
        _case("attach_within400", kind="attach", within=400.0, vessels=50, per_vessel=200),
        # a burst of kNN and within requests of mixed sizes to the server
        _case("serve_burst", kind="serve", vessels=100, requests=20, most=1000),
        # the refine seam on host arrays, voxel pairs of ragged sizes
        _case("refine_batch", kind="refine", pairs=3000, most=130, form=1),
        # LOD preparation of many small objects, and of few large ones
        _case("prep_nuclei", kind="prep", which="nuclei", vessels=8, per_vessel=125, voxel_size=100),
        _case("prep_vessels", kind="prep", which="vessels", vessels=6, per_vessel=1, voxel_size=100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["join"] * 8 + ["attach", "serve", "refine", "prep"])
    if kind in ("join", "attach"):
        form = rng.choice(["nn", "nn_self", "within", "within", "within_self", "exact"] if kind == "join" else ["nn", "within"])
        knn = _log(rng, 1, 30)
        per = _log(rng, 7, 150)
        c = dict(vessels=_log(rng, 10, 90), per_vessel=per, subdiv=rng.choice([2, 3, 3]), voxel_size=rng.randint(50, 150),
                 level=rng.choice([0, 1, 2, 2, 2, 2]), lods=rng.choice(["", "", "", "20,60,100", "100"]), kind=kind)
        if form == "nn":
            c.update(query="nn", knn=min(knn, c["vessels"] - 1))
        elif form == "nn_self":
            c.update(query="nn", knn=min(knn, 20), self=True, vessels=_log(rng, 2, 16))
        elif form == "within":
            c.update(within=round(rng.uniform(50.0, 800.0), 1))
        elif form == "within_self":
            c.update(within=round(rng.uniform(10.0, 80.0), 1), self=True)
        else:
            c.update(within=round(rng.uniform(50.0, 250.0), 1), exact=True, vessels=_log(rng, 10, 50), per_vessel=_log(rng, 7, 30))
        return _case(None, **c)
    if kind == "serve":
        return _case(None, kind="serve", vessels=_log(rng, 20, 100), requests=rng.randint(3, 20), most=_log(rng, 50, 1000))
    if kind == "refine":
        return _case(None, kind="refine", pairs=_log(rng, 50, 3000), most=rng.randint(20, 130), form=1)
    if rng.random() < 0.7:
        return _case(None, kind="prep", which="nuclei", vessels=_log(rng, 1, 8), per_vessel=_log(rng, 10, 120),
                     voxel_size=rng.randint(60, 150))
    return _case(None, kind="prep", which="vessels", vessels=rng.randint(1, 6), per_vessel=1, voxel_size=rng.randint(60, 150))


# ---- inputs ----------------------------------------------------------------

_contexts = {}


def _context(role):
    """The process's context for one role, made once: tiles come and go, the context stays."""
    if role not in _contexts:
        _contexts[role] = tdp.Context(0)
    return _contexts[role]


def _gen(case):
    kw = {"voxel_size": case.get("voxel_size", 100), "nucleus_subdiv": case.get("subdiv", 3)}
    return case["vessels"], case["per_vessel"], kw


def _join_args(case):
    a = {"query": case["query"], "hausdorff_level": case["level"], "exact_distances": case["exact"]}
    if case["query"] == "nn":
        a["knn"] = case["knn"]
    else:
        a["within"] = case["within"]
    if case["lods"]:
        a["lods"] = [int(x) for x in case["lods"].split(",")]
    return a


def _voxel_pairs(case, seed):
    """Facing patches of triangles, up to `most` a side, with the Hausdorff pairs an LOD would have."""
    rng = np.random.default_rng(seed)
    n = np.stack([rng.integers(1, case["most"] + 1, case["pairs"]), rng.integers(1, case["most"] + 1, case["pairs"])], 1)
    counts = n.reshape(-1)
    ends = np.cumsum(counts)
    starts = ends - counts
    voxel = np.repeat(np.arange(2 * case["pairs"]), counts)
    gap = rng.uniform(5.0, 60.0, case["pairs"])
    way = rng.normal(size=(case["pairs"], 3))
    way /= np.linalg.norm(way, axis=1, keepdims=True)
    at = rng.uniform(0.0, 1000.0, (case["pairs"], 3))
    centre = np.stack([at, at + gap[:, None] * way], 1).reshape(-1, 3)
    c = centre[voxel] + rng.uniform(-6.0, 6.0, (len(voxel), 3))
    tri = (c[:, None, :] + rng.normal(size=(len(voxel), 3, 3))).reshape(-1, 9).astype(np.float32)
    hd = (np.abs(rng.normal(size=(len(voxel), 2))) * 0.2).astype(np.float32)
    rows = np.stack([starts[0::2], n[:, 0], starts[1::2], n[:, 1]], 1).astype(np.uint64)
    return tri, hd, rows


def _requests(case):
    """(nuclei, query, k, tau) of each request: log-uniform sizes, 60 % kNN, 40 % within."""
    rng = np.random.default_rng(case["requests"] * 1009 + case["most"])
    out = []
    for _ in range(case["requests"]):
        n = int(round(math.exp(rng.uniform(0.0, math.log(case["most"])))))
        nn = rng.random() < 0.6
        out.append((n, "nn" if nn else "within", int(rng.integers(1, min(50, case["vessels"] - 1) + 1)), float(rng.uniform(50.0, 800.0))))
    return out


def _rows(n, targets, query, knn, own):
    """Result arrays that a program keeps for a join of n queries: more rows than such a join has
    (a within query of this workload reports a few vessels, or some tens of its neighbours)."""
    cap = n * (min(knn, targets) if query == "nn" else min(targets, 128 if own else 20))
    return {"q": np.full(cap, -1, np.int32), "t": np.full(cap, -1, np.int32), "d": None, "n": 0}


def _keep(rows, got):
    """A join's result into the program's arrays; rows past the last one read -1 (ids) and 0 (distances)."""
    q, t, d = got
    n = len(q)
    if rows["d"] is None:
        rows["d"] = np.zeros(len(rows["q"]), d.dtype)
    for name, values, empty in (("q", q, -1), ("t", t, -1), ("d", d, 0)):
        rows[name][:n] = values
        rows[name][n:rows["n"]] = empty
    rows["n"] = n
    return rows["q"], rows["t"], rows["d"]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("join", "attach"):
        nv, npv, kw = _gen(case)
        nb, vb = tdp.gen_tiles(nv, npv, seed=seed, only="nuclei" if case["self"] else None, **kw)
        ctx = s["ctx"] = _context(("autotuned" if case["autotune"] else "default") + " " + kind)
        s["args"] = _join_args(case)
        targets = nv * npv - 1 if case["self"] else nv
        s["rows"] = _rows(nv * npv, targets, case["query"], case["knn"], case["self"])
        if kind == "join":
            s["t1"] = tdp.Tile(ctx, nb)
            s["t2"] = None if case["self"] else tdp.Tile(ctx, vb)
            if case["autotune"]:  # once per kind of join, as a program does when it starts
                ctx.autotune(s["t1"], s["t2"], query=case["query"], knn=max(case["knn"], 1), within=case["within"])
        else:
            s["b1"], s["b2"] = tdp.pinned_copy(nb), tdp.pinned_copy(vb)
    elif kind == "serve":
        nb, vb = tdp.gen_tiles(case["vessels"], max(1, -(-case["most"] // case["vessels"])), seed=seed)
        ctx = s["ctx"] = tdp.Context(0)
        s["tile"] = tdp.Tile(ctx, vb)
        off = tdp.raw_object_offsets(nb)
        rng = np.random.default_rng(seed + 2)
        s["requests"], s["rows"] = [], []
        for n, q, k, tau in _requests(case):
            b = int(rng.integers(0, len(off) - n))
            s["requests"].append((tdp.pinned_copy(tdp.raw_slice(nb, off, b, b + n)), q, k, tau))
            s["rows"].append(_rows(n, case["vessels"], q, k, False))
        s["server"] = tdp.Server(ctx, s["tile"], arena_objects=1 << 14, arena_voxels=1 << 18, arena_tris=1 << 24)
    elif kind == "refine":
        s["ctx"] = _context("refine")
        s["batch"] = _voxel_pairs(case, seed)
    else:
        s["ctx"] = _context("prep")
        s["mesh"] = tdp.gen_meshes(case["vessels"], case["per_vessel"], seed=seed, which=case["which"])
        s["out"] = np.zeros(tdp.raw_prep_bound(s["mesh"][3], case["voxel_size"]), np.uint8)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "join":
        return _keep(s["rows"], s["ctx"].join(s["t1"], s["t2"], **s["args"]))
    if kind == "attach":
        t1 = tdp.Tile(s["ctx"], s["b1"], attach=True)
        t2 = tdp.Tile(s["ctx"], s["b2"], attach=True)
        out = s["ctx"].join(t1, t2, **s["args"])
        t1.free()
        t2.free()
        return _keep(s["rows"], out)
    if kind == "serve":
        ids = [s["server"].submit(raw, query=q, knn=k, within=tau) for raw, q, k, tau in s["requests"]]
        return [_keep(rows, s["server"].wait(i)[:3]) for rows, i in zip(s["rows"], ids)]
    if kind == "refine":
        return s["ctx"].refine_batch(*s["batch"], form=case["form"])
    tile, _ = s["ctx"].raw_from_meshes(*s["mesh"], voxel_size=case["voxel_size"], out=s["out"])
    return s["out"], tile.size


# ---- what a pass cannot do without -------------------------------------------

def _sizes(case):
    """(nuclei, their triangles, vessels, their triangles) of the workload."""
    n = case["vessels"] * case.get("per_vessel", 1)
    return n, n * 20 * 4 ** case.get("subdiv", 3), case["vessels"], case["vessels"] * 20000


def work(case):
    kind = case["kind"]
    if kind == "refine":
        # every triangle (9 + 2 floats) and row in, three floats a pair out; one
        # distance a voxel pair at the least
        tris = case["pairs"] * (case["most"] + 1)
        return {"bytes": tris * 44 + case["pairs"] * 44, "flops": case["pairs"] * 966}
    n, nt, v, vt = _sizes(case)
    if kind == "prep":
        # vertices and facets in, five LODs of 44-byte triangles out
        t = nt if case["which"] == "nuclei" else vt
        return {"bytes": t * 18 + t * 3 * 44, "flops": t * 1000}
    if kind == "serve":
        sizes = sum(r[0] for r in _requests(case))
        return {"bytes": (sizes * 13 + vt // 100) * 36 + sizes * 12 * 10, "flops": sizes * 10 * 966}
    # a join reads every voxel record (box and core, 36 bytes) and object box
    # once and writes 12 bytes a result; which triangles it has to read depends
    # on the data: one voxel pair of about 100 triangles a side for each result,
    # up to every LOD-100 triangle of both tiles
    rows = n * (case["knn"] if case["query"] == "nn" else max(1.0, (case["within"] / 400.0) ** 2))
    per = case["voxel_size"]
    vox = (nt + (0 if case["self"] else vt)) / per
    tris = min(rows * 2 * per, nt + (0 if case["self"] else vt))
    per_row = 966 * (10 if case["exact"] else 1)
    return {"bytes": vox * 36 + (n + v) * 36 + rows * 12 + tris * 44, "flops": rows * per_row}


# ---- 64-bit values, without the package's code -------------------------------

def _seg_seg(p, d, q, e):
    """Squared distance of segments p + s d and q + t e (any batch), by the least of the
    interior solution and the four end points against the other segment."""
    def end(x, a, w):
        ww = (w * w).sum(-1).clamp_min(1e-300)
        t = (((x - a) * w).sum(-1) / ww).clamp(0.0, 1.0)
        r = x - a - t[..., None] * w
        return (r * r).sum(-1)

    best = torch.minimum(torch.minimum(end(p, q, e), end(p + d, q, e)), torch.minimum(end(q, p, d), end(q + e, p, d)))
    r = p - q
    a, b, c = (d * d).sum(-1), (d * e).sum(-1), (e * e).sum(-1)
    f, g = (d * r).sum(-1), (e * r).sum(-1)
    den = a * c - b * b
    ok = den > 1e-14 * a * c
    den = torch.where(ok, den, torch.ones_like(den))
    s, t = (b * g - c * f) / den, (a * g - b * f) / den
    ok &= (s > 0) & (s < 1) & (t > 0) & (t < 1)
    w = r + s[..., None] * d - t[..., None] * e
    return torch.where(ok, torch.minimum(best, (w * w).sum(-1)), best)


def _tri_tri(A, B):
    """Distances of triangles A[i] and B[i] (n x 3 x 3 doubles); 0 where they meet."""
    best = torch.full(A.shape[:1], 1e300, dtype=A.dtype, device=A.device)
    for i in range(3):
        for j in range(3):
            best = torch.minimum(best, _seg_seg(A[:, i], A[:, (i + 1) % 3] - A[:, i], B[:, j], B[:, (j + 1) % 3] - B[:, j]))
    meet = torch.zeros_like(best, dtype=torch.bool)
    for F, G in ((A, B), (B, A)):
        n = torch.linalg.cross(F[:, 1] - F[:, 0], F[:, 2] - F[:, 0])
        nn = (n * n).sum(-1)

        def inside(x):
            ok = nn > 0
            for k in range(3):
                w = torch.linalg.cross(n, F[:, (k + 1) % 3] - F[:, k])
                ok = ok & (((x - F[:, k]) * w).sum(-1) >= 0)
            return ok

        h = ((G - F[:, None, 0]) * n[:, None]).sum(-1)
        for k in range(3):
            best = torch.where(inside(G[:, k]), torch.minimum(best, h[:, k] ** 2 / nn.clamp_min(1e-300)), best)
            a, b = h[:, k], h[:, (k + 1) % 3]
            cross = a * b < 0
            t = torch.where(cross, a / torch.where(cross, a - b, torch.ones_like(a)), torch.zeros_like(a))
            meet |= cross & inside(G[:, k] + t[:, None] * (G[:, (k + 1) % 3] - G[:, k]))
    return torch.where(meet, torch.zeros_like(best), best).sqrt()


def _exact_refine(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    tri, hd, rows = _voxel_pairs(case, seed)
    T = torch.from_numpy(tri.astype(np.float64)).reshape(-1, 3, 3).to(dev)
    H = torch.from_numpy(hd.astype(np.float64)).to(dev)
    out = torch.empty((len(rows), 3), dtype=torch.float64)
    for i, (o1, n1, o2, n2) in enumerate(rows.astype(np.int64).tolist()):
        a = torch.arange(o1, o1 + n1, device=dev).repeat_interleave(n2)
        b = torch.arange(o2, o2 + n2, device=dev).repeat(n1)
        d = _tri_tri(T[a], T[b])
        lo = (d - H[a, 0] - H[b, 0]).clamp_min(0.0)
        out[i, 0], out[i, 1], out[i, 2] = d.min(), lo.min(), (d + H[a, 1] + H[b, 1]).min()
    return out.numpy()


def _exact_within(case, seed):
    """Every (nucleus, vessel) pair within tau with its distance, by query then result."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    nv, npv, kw = _gen(case)
    sides = []
    for which in ("nuclei", "vessels"):
        V, vo, F, fo = tdp.gen_meshes(nv, npv, seed=seed, which=which, **kw)
        tris = [torch.from_numpy(V[vo[o]:vo[o + 1]].astype(np.float64)[F[fo[o]:fo[o + 1]]]).to(dev) for o in range(len(vo) - 1)]
        c = [t.mean(1) for t in tris]
        r = [(t - m[:, None]).norm(dim=2).amax(1) for t, m in zip(tris, c)]
        lo = torch.stack([t.reshape(-1, 3).amin(0) for t in tris]).cpu()
        hi = torch.stack([t.reshape(-1, 3).amax(0) for t in tris]).cpu()
        sides.append((tris, c, r, lo, hi))
    (A, cA, rA, loA, hiA), (B, cB, rB, loB, hiB) = sides
    found = []
    for i in range(len(A)):
        gap = torch.maximum(torch.maximum(loB - hiA[i], loA[i] - hiB), torch.zeros(3, dtype=torch.float64)).norm(dim=1)
        mid = cA[i].mean(0)
        rad = ((cA[i] - mid).norm(dim=1) + rA[i]).max()
        for j in torch.nonzero(gap <= case["within"] * 1.001).flatten().tolist():
            near = (cB[j] - mid).norm(dim=1) - rB[j]  # a vessel triangle's least distance from the nucleus' centre
            k = torch.nonzero(near <= (near + 2 * rB[j]).min() + 2 * rad).flatten()
            sep = torch.cdist(cA[i], cB[j][k], compute_mode="donot_use_mm_for_euclid_dist")
            a, b = torch.nonzero(sep - rA[i][:, None] - rB[j][k][None] <= sep.min(), as_tuple=True)
            d = float(_tri_tri(A[i][a], B[j][k][b]).min())
            if d <= case["within"]:
                found.append((i, j, d))
    out = np.zeros(len(_rows(nv * npv, nv, "within", 0, False)["q"]), np.float64)
    out[:len(found)] = [f[2] for f in sorted(found)]
    return out


def exact(case, seed):
    """FP64 values where a pass returns distances that have one: the refine's three minima, and the exact-distance join's."""
    if case["kind"] == "refine":
        return _exact_refine(case, seed)
    # the FP32 bounds of the other joins depend on the LOD that decided a pair
    if case["kind"] == "join" and case["exact"] and case["query"] == "within" and not case["self"] and case["vessels"] * case["per_vessel"] <= 1000:
        return None, None, _exact_within(case, seed)
    return None
