"""Measured cases: the work a program has the tessellator do, through its public entry points.

A program that moves particles replaces the points of a diagram, computes every cell and takes volumes, neighbour
lists and face areas out of it (kind "diagram", from device memory; kind "host", from and to host arrays); it does
the same for many small diagrams at once (kind "batch"); it asks for one cell with a container of its own (kind
"cell") and for the neighbours of many positions within a radius (kind "radius").

Results of the FP32 + guard form are good to about 1e-7, so the program keeps them as float32; those of the FP64 and
MIXED forms stay float64.  The library's result buffers are valid until the next compute, so results are copied out,
into arrays of the program's own that have room for any input of that size (what lies beyond a result stays 0).
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "the-tessellator_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import tessellator as T  # noqa: E402

DEV = "cuda"
#: Values of a cell and its faces: about 15.5 faces a cell for random points.
FACES = 15.5
#: Faces of a cell at most, and room for the faces of n cells.
MOST_FACES = 254
#: FP operations of a cell (12 per bisector, 6 per vertex test, 13 per new vertex, 12 per fan triangle, 3 per face).
CELL_FLOPS = 9500


def _diagram(name, n, precision, points="uniform", box=(1.0, 1.0, 1.0), groups=0):
    """groups > 0: every point carries a group id below it, and cells are cut by the points of group 0 alone."""
    return {"name": name, "kind": "diagram", "n": n, "precision": precision, "points": points,
            "bx": box[0], "by": box[1], "bz": box[2], "groups": groups}


def listed():
    return [
        # one cell asked for by its index, its container given with the call (Diagram::get_cell_at_index): latency
        {"name": "one_cell_of_1000", "kind": "cell", "n": 1000, "precision": "fp64"},
        # the smallest whole diagram: launches and host work
        _diagram("uniform_1000_fp32", 1000, "fp32"),
        # the plain FP64 tessellation of 10,000 points in the unit cube
        _diagram("uniform_10000_fp64", 10_000, "fp64"),
        # an ordinary step with host arrays in and out: upload, binning, cells, read-back
        {"name": "host_60000_mixed", "kind": "host", "n": 60_000, "precision": "mixed"},
        # two species, cells against one of them only; an odd count in an oblong box, FP64-accurate volumes
        _diagram("two_species_99991_mixed", 99_991, "mixed", box=(2.0, 1.0, 0.5), groups=2),
        # plain FP64 at a size that fills the GPU
        _diagram("uniform_250007_fp64", 250_007, "fp64"),
        # a million uniform points, the ordinary large diagram
        _diagram("uniform_1000000_fp32", 1_000_000, "fp32"),
        # a crystal with thermal motion (simple cubic, spacing 1): near-degenerate vertices, guard-band re-runs
        _diagram("crystal_96_fp32", 96 ** 3, "fp32", points="crystal", box=(96.0, 96.0, 96.0)),
        # clustered points (galaxies, droplets): uneven neighbour counts and crowded bins
        _diagram("clustered_2097152_fp32", 2_097_152, "fp32", points="clustered", box=(100.0, 100.0, 100.0)),
        # many independent diagrams of 64 to 16,384 points, each in its own box, in one graph launch
        {"name": "batch_768_fp32", "kind": "batch", "ndiag": 768, "nmin": 64, "nmax": 16_384, "precision": "fp32"},
        # neighbours within a radius of a million positions (about 16 results each), as a particle code asks every step
        {"name": "radius_1000000", "kind": "radius", "n": 1_000_000, "nq": 1_000_000, "mean": 16.0},
        # the largest: 16,777,216 points, one per unit of volume
        _diagram("uniform_16777216_fp32", 16_777_216, "fp32", box=(256.0, 256.0, 256.0)),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["diagram"] * 5 + ["host", "batch", "radius", "cell"])
    precision = rng.choice(["fp32", "fp32", "mixed", "fp64"])
    if kind == "cell":
        return {"kind": "cell", "n": _log(rng, 200, 100_000), "precision": precision}
    if kind == "host":
        return {"kind": "host", "n": _log(rng, 500, 300_000), "precision": "mixed" if precision == "fp32" else precision}
    if kind == "batch":
        return {"kind": "batch", "ndiag": _log(rng, 8, 1024), "nmin": 64, "nmax": _log(rng, 256, 16_384),
                "precision": precision}
    if kind == "radius":
        return {"kind": "radius", "n": _log(rng, 5000, 2_000_000), "nq": _log(rng, 1000, 2_000_000),
                "mean": rng.choice([6.0, 16.0, 40.0])}
    points = rng.choice(["uniform", "uniform", "clustered", "crystal"])
    if points == "crystal":
        m = _log(rng, 12, 110)
        c = _diagram("", m ** 3, "fp32" if precision == "fp64" else precision, points, (float(m),) * 3)
    elif points == "clustered":
        c = _diagram("", _log(rng, 3000, 2_000_000 if precision != "fp64" else 500_000), precision, points, (100.0,) * 3)
    else:
        n = _log(rng, 300, 4_000_000 if precision != "fp64" else 1_000_000)
        side = rng.choice([1.0, 8.0, 100.0])
        c = _diagram("", n, precision, points, (side, side * rng.choice([1.0, 0.7]), side * rng.choice([1.0, 1.5])),
                     rng.choice([0, 0, 2]))
    del c["name"]
    return c


# ---- inputs ----
def _points(case, gen):
    """n x 3 doubles on the GPU, inside the box."""
    n = case["n"]
    side = torch.tensor([case["bx"], case["by"], case["bz"]], dtype=torch.float64, device=DEV)
    rand = lambda *s: torch.rand(*s, generator=gen, dtype=torch.float64, device=DEV)  # noqa: E731
    if case["points"] == "uniform":
        return rand(n, 3) * side
    if case["points"] == "crystal":
        m = round(n ** (1.0 / 3.0))
        g = torch.arange(m, dtype=torch.float64, device=DEV) + 0.5
        p = torch.stack(torch.meshgrid(g, g, g, indexing="ij"), dim=-1).reshape(-1, 3)
        return p + (rand(n, 3) - 0.5) * 2e-3    # thermal motion, a thousandth of the spacing
    # clustered: 90% in 64 Gaussians of sigma 0.01 of the box, 10% uniform; draws outside are taken again
    nb = int(round(0.1 * n))
    centres = 0.1 + 0.8 * rand(64, 3)
    which = torch.randint(0, 64, (n - nb,), generator=gen, device=DEV)
    p = centres[which] + 0.01 * torch.randn(n - nb, 3, generator=gen, dtype=torch.float64, device=DEV)
    for _ in range(4):
        out = ((p < 0.0) | (p >= 1.0)).any(dim=1, keepdim=True)
        p = torch.where(out, centres[which] + 0.01 * torch.randn(n - nb, 3, generator=gen, dtype=torch.float64, device=DEV), p)
    p = torch.cat([p.clamp(0.0, 1.0 - 1e-9), rand(nb, 3)])
    return p[torch.randperm(n, generator=gen, device=DEV)] * side


def _groups(case, gen):
    if not case["groups"]:
        return None
    return torch.randint(0, case["groups"], (case["n"],), generator=gen, device=DEV)


def _batch(case, gen):
    """(points on the GPU, offsets, boxes): sizes log-uniform (the same for every seed), sides uniform in [0.5, 2]."""
    sizes = np.random.RandomState(17).rand(case["ndiag"])
    sizes = np.rint(np.exp(np.log(case["nmin"]) + sizes * np.log(case["nmax"] / case["nmin"]))).astype(np.int64)
    sides = 0.5 + 1.5 * torch.rand(case["ndiag"], 3, generator=gen, dtype=torch.float64, device=DEV).cpu().numpy()
    offs = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    scale = torch.from_numpy(np.repeat(sides, sizes, axis=0)).to(DEV)
    pts = torch.rand(int(offs[-1]), 3, generator=gen, dtype=torch.float64, device=DEV) * scale
    return pts, offs, np.concatenate([np.zeros_like(sides), sides], axis=1)


def _room(n):
    return 18 * n + 1024


def _radius_of(case):
    return (case["mean"] * 3.0 / (4.0 * math.pi * case["n"])) ** (1.0 / 3.0)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _inputs(case, seed):
    """What exact() and prepare() share: the numbers that the seed makes."""
    gen = _gen(seed)
    kind = case["kind"]
    if kind in ("diagram", "host", "cell"):
        full = case if kind == "diagram" else dict(case, points="uniform", bx=1.0, by=1.0, bz=1.0, groups=0)
        pts = _points(full, gen)
        return {"points": pts, "groups": _groups(full, gen), "box": [full["bx"], full["by"], full["bz"]],
                "index": int(seed) * 7919 % case["n"]}
    if kind == "batch":
        pts, offs, boxes = _batch(case, gen)
        return {"points": pts, "offsets": offs, "boxes": boxes}
    return {"points": torch.rand(case["n"], 3, generator=gen, dtype=torch.float64, device=DEV),
            "queries": torch.rand(case["nq"], 3, generator=gen, dtype=torch.float64, device=DEV)}


def prepare(case, seed):
    inp = _inputs(case, seed)
    state = dict(inp, kind=case["kind"], precision=case.get("precision"))
    # the library runs on the program's own stream, so that its results can be read there in order
    state["stream"] = stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    cfg = T.default_config(stream=stream.cuda_stream)
    n = len(inp["points"])
    if case["kind"] in ("diagram", "batch"):
        kept = torch.float32 if case["precision"] == "fp32" else torch.float64
        state["out"] = {"volumes": torch.zeros(n, dtype=kept, device=DEV),
                        "offsets": torch.zeros(n + 1, dtype=torch.int64, device=DEV),
                        "neighbors": torch.zeros(_room(n), dtype=torch.int32, device=DEV),
                        "areas": torch.zeros(_room(n), dtype=kept, device=DEV)}
    if case["kind"] == "batch":
        torch.cuda.synchronize()
        state["batch"] = T.Batch(inp["points"].cpu().numpy(), inp["offsets"], inp["boxes"], config=cfg)
        return state
    box = inp.get("box", [1.0, 1.0, 1.0])
    g = inp.get("groups")
    state["diagram"] = T.Diagram(groups=None if g is None else g.to(torch.int32).cpu().numpy().astype(np.uint32),
                                 container=T.Polyhedron(0.0, 0.0, 0.0, *box), config=cfg,
                                 device_ptr=inp["points"].data_ptr(), n=n)
    if case["kind"] == "host":       # pinned arrays, as a program keeps them for its transfers
        state["host_points"] = T.pinned_empty(3 * n, np.float64)
        state["host_points"][:] = inp["points"].cpu().numpy().reshape(-1)
        state["out"] = {"volumes": T.pinned_empty(n, np.float64), "offsets": T.pinned_empty(n + 1, np.uint64),
                        "neighbors": T.pinned_empty(_room(n), np.int32), "areas": T.pinned_empty(_room(n), np.float64)}
        for a in state["out"].values():
            a[:] = 0
    if case["kind"] == "radius":
        state["r"] = _radius_of(case)
        state["cap"] = int(case["nq"] * case["mean"] * 1.3) + 4096
        state["offs"] = torch.zeros(case["nq"] + 1, dtype=torch.int64, device=DEV)
        state["ids"] = torch.zeros(state["cap"], dtype=torch.int32, device=DEV)
    torch.cuda.synchronize()
    return state


# ---- one pass ----
def _device_results(owner, n, out):
    """Copies of the results in device memory (float32 for the FP32 form, float64 for the others)."""
    v, o, nb, a, total = owner.results_device()
    view = lambda p, k, t: torch.as_tensor(T.DeviceArray(p, k, t), device=DEV)  # noqa: E731
    out["volumes"].copy_(view(v, n, np.float64))
    out["offsets"].copy_(view(o, n + 1, np.uint64).view(torch.int64))
    out["neighbors"][:total].copy_(view(nb, total, np.int32))
    out["areas"][:total].copy_(view(a, total, np.float64))
    return out


def _check(status):
    if status != 0:
        raise T.TessError(status, T.last_error())


def run(state):
    kind = state["kind"]
    with torch.cuda.stream(state["stream"]):
        if kind == "diagram":
            d = state["diagram"]
            d.update_points(device_ptr=state["points"].data_ptr())
            d.compute_all(state["precision"], target_group=None if state["groups"] is None else 0)
            return _device_results(d, d.n, state["out"])
        if kind == "batch":
            b = state["batch"]
            b.update_points(device_ptr=state["points"].data_ptr())
            b.compute(state["precision"])
            return _device_results(b, b.n, state["out"])
        if kind == "host":
            d = state["diagram"]
            d.update_points(state["host_points"])
            d.compute_all(state["precision"])
            out, total = state["out"], ctypes.c_size_t(0)
            at = lambda name, t: out[name].ctypes.data_as(ctypes.POINTER(t))  # noqa: E731
            _check(T.lib().tess_volumes(d._h, at("volumes", ctypes.c_double)))
            _check(T.lib().tess_neighbors_csr(d._h, at("offsets", ctypes.c_uint64), at("neighbors", ctypes.c_int32),
                                              at("areas", ctypes.c_double), len(out["areas"]), ctypes.byref(total)))
            return dict(out, offsets=out["offsets"].view(np.int64))
        if kind == "cell":
            c = state["diagram"].get_cell_at_index(state["index"], T.Polyhedron(0.0, 0.0, 0.0, 1.0, 1.0, 1.0),
                                                   precision=state["precision"]).compute_voronoi_cell()
            kept = np.float32 if state["precision"] == "fp32" else np.float64
            nbr, area = np.zeros(MOST_FACES, dtype=np.int32), np.zeros(MOST_FACES, dtype=kept)
            ids, faces = c.compute_neighbors(), c.compute_faces()
            nbr[:len(ids)] = ids
            area[:len(faces)] = [f.compute_area() for f in faces]
            return {"volumes": np.array([c.compute_volume()], dtype=kept), "neighbors": nbr, "areas": area}
        total = ctypes.c_size_t(0)
        q = state["queries"]
        _check(T.lib().tess_find_neighbors_in_radius(state["diagram"]._h, q.data_ptr(), len(q), state["r"], 1, 1,
                                                     state["offs"].data_ptr(), state["ids"].data_ptr(), state["cap"],
                                                     ctypes.byref(total)))
        return {"offsets": state["offs"], "ids": state["ids"]}


def _total_points(case):
    if case["kind"] != "batch":
        return case["n"]
    lo, hi = case["nmin"], case["nmax"]
    return case["ndiag"] * (hi - lo) / math.log(hi / lo) if hi > lo else case["ndiag"] * lo


def work(case):
    if case["kind"] == "radius":
        # 24 B a query and an offset of 8 B; the points in reach once each (24 B); 4 B a result
        return {"bytes": case["nq"] * (24 + 8 + 4 * case["mean"]) + 24 * case["n"],
                "flops": 8 * case["nq"] * case["mean"] * 27 / (4.0 * math.pi / 3.0)}
    if case["kind"] == "cell":
        return {"bytes": 24 * 64 + 8 + 12 * FACES, "flops": CELL_FLOPS}
    n = _total_points(case)
    return {"bytes": n * (24 + 8 + 8 + 12 * FACES), "flops": n * CELL_FLOPS}


# ---- the same in 64 bits, without the library ----
def _half_spaces(nrm, off, ok):
    """Faces of the polytopes {x : nrm . x <= off} (c x p planes, `ok` marks the real ones): area of each face,
    volume (the origin inside), and the end points of every edge with a mask.  Each pair of planes meets in a line,
    which the other planes clip to the edge."""
    c, p = off.shape
    i, j = torch.triu_indices(p, p, 1, device=off.device)
    ni, nj, hi, hj = nrm[:, i], nrm[:, j], off[:, i, None], off[:, j, None]
    u = torch.linalg.cross(ni, nj)
    uu = (u * u).sum(-1, keepdim=True)
    scale = (ni * ni).sum(-1, keepdim=True) * (nj * nj).sum(-1, keepdim=True)
    live = (uu[..., 0] > 1e-24 * scale[..., 0]) & ok[:, i] & ok[:, j]
    safe = torch.where(live[..., None], uu, torch.ones_like(uu))
    p0 = (hi * torch.linalg.cross(nj, u) + hj * torch.linalg.cross(u, ni)) / safe
    lo = torch.full_like(safe[..., 0], -math.inf)
    hi_t = torch.full_like(lo, math.inf)
    for k in range(p):
        nk = nrm[:, k, None]
        a = (nk * u).sum(-1)
        b = off[:, k, None] - (nk * p0).sum(-1)
        use = ok[:, k, None] & (i != k) & (j != k)
        t = b / torch.where(a == 0, torch.ones_like(a), a)
        hi_t = torch.where(use & (a > 0), torch.minimum(hi_t, t), hi_t)
        lo = torch.where(use & (a < 0), torch.maximum(lo, t), lo)
        live = live & ~(use & (a == 0) & (b < 0))
    live = live & (hi_t > lo) & torch.isfinite(hi_t) & torch.isfinite(lo)
    lo, hi_t = torch.where(live, lo, torch.zeros_like(lo)), torch.where(live, hi_t, torch.zeros_like(lo))
    length = (hi_t - lo) * safe[..., 0].sqrt() * live
    area = torch.zeros_like(off)
    for a, b in ((i, j), (j, i)):      # a triangle from the foot of plane a's normal to the edge with plane b
        na, nb, ha, hb = nrm[:, a], nrm[:, b], off[:, a], off[:, b]
        n2 = (na * na).sum(-1)
        foot = na * (ha / n2)[..., None]
        inward = nb - na * ((na * nb).sum(-1) / n2)[..., None]
        dist = (hb - (nb * foot).sum(-1)) / inward.norm(dim=-1).clamp_min(1e-300)
        area.scatter_add_(1, a.expand(c, -1), 0.5 * dist * length)
    height = off / nrm.norm(dim=-1).clamp_min(1e-300)
    volume = (area * torch.where(ok, height, torch.zeros_like(height))).sum(-1) / 3.0
    seen = torch.zeros_like(off)
    for a in (i, j):
        seen.scatter_add_(1, a.expand(c, -1), live.to(off.dtype))
    ends = torch.cat([p0 + lo[..., None] * u, p0 + hi_t[..., None] * u], dim=1)
    return area, volume, seen >= 3, ends, torch.cat([live, live], dim=1)


def _cells(sites, own, pool, ids, box):
    """(volume, face count, areas sorted by neighbour id as one list) of the cells of `sites` against the points
    `pool` (their ids: `ids`), walls at 0 and box; `own`: the sites' own ids.  The nearest points first; a farther
    one joins where it cuts a vertex, until none does."""
    k = min(len(pool), 1024)
    dist = torch.cdist(sites, pool, compute_mode="donot_use_mm_for_euclid_dist")
    dist = torch.where(own[:, None] == ids[None, :], torch.full_like(dist, math.inf), dist)
    near, at = dist.topk(k, dim=1, largest=False)
    rel = pool[at] - sites[:, None]
    cid = ids[at]
    valid = torch.isfinite(near)
    half = 0.5 * (rel * rel).sum(-1)
    eye = torch.eye(3, dtype=torch.float64, device=DEV)
    wall_n = torch.stack([-eye, eye], dim=1).reshape(6, 3).expand(len(sites), 6, 3)
    wall_h = torch.stack([sites, box - sites], dim=2).reshape(-1, 6)
    wall_id = torch.arange(-1, -7, -1, device=DEV).expand(len(sites), 6)
    inside = torch.zeros_like(valid)
    inside[:, :24] = True
    inside &= valid
    for _ in range(200):
        take = int(inside.sum(1).max())
        order = torch.argsort((~inside).to(torch.int8), dim=1, stable=True)[:, :take]
        ok = torch.cat([torch.ones_like(wall_h, dtype=torch.bool), inside.gather(1, order)], dim=1)
        nrm = torch.cat([wall_n, rel.gather(1, order[..., None].expand(-1, -1, 3))], dim=1)
        off = torch.cat([wall_h, half.gather(1, order)], dim=1)
        who = torch.cat([wall_id, cid.gather(1, order)], dim=1)
        nrm = torch.where(ok[..., None], nrm, torch.ones_like(nrm))
        area, volume, face, ends, live = _half_spaces(nrm, off, ok)
        # the farthest-cutting twelve of the points whose plane some vertex lies beyond
        most = torch.full_like(half, -math.inf)
        count = live.sum(1).max()
        pick = torch.argsort((~live).to(torch.int8), dim=1, stable=True)[:, :int(count)]
        v = ends.gather(1, pick[..., None].expand(-1, -1, 3))
        lv = live.gather(1, pick)
        reach = torch.where(lv, v.norm(dim=-1), torch.zeros_like(lv, dtype=torch.float64)).amax(1)
        for q in range(0, v.shape[1], 16):
            s = torch.einsum("cvx,ckx->ckv", v[:, q:q + 16], rel) - half[..., None]
            s = torch.where(lv[:, None, q:q + 16], s, torch.full_like(s, -math.inf))
            most = torch.maximum(most, s.amax(-1))
        cuts = valid & ~inside & (most > 1e-14 * half)
        if not bool(cuts.any()):
            break
        keep = torch.zeros_like(inside).scatter_(1, order, face[:, 6:] & inside.gather(1, order))
        first = (cuts.cumsum(1) <= 12) & cuts
        inside = keep | first
    else:
        return None
    if k < len(pool) and bool((2.0 * reach > near[:, -1]).any()):
        return None
    who = torch.where(face, who, torch.full_like(who, 1 << 60))
    order = torch.argsort(who, dim=1)
    return volume, face.sum(1), area.gather(1, order)[face.gather(1, order)]


def exact(case, seed):
    """Volumes and areas of small diagrams and of single cells in 64 bits (larger ones take too long)."""
    kind = case["kind"]
    if kind not in ("diagram", "host", "cell") or case["n"] > 120_000:
        return None
    inp = _inputs(case, seed)
    pts, box = inp["points"], torch.tensor(inp["box"], dtype=torch.float64, device=DEV)
    ids = torch.arange(len(pts), device=DEV)
    pool = ids if inp["groups"] is None else ids[inp["groups"] == 0]
    own = ids if kind != "cell" else ids[inp["index"]:inp["index"] + 1]
    parts = []
    for b in range(0, len(own), 1024):
        sites = own[b:b + 1024]
        got = _cells(pts[sites], sites, pts[pool], pool, box)
        if got is None:
            return None
        parts.append(got)
    areas = torch.cat([p[2] for p in parts])
    room = torch.zeros(MOST_FACES if kind == "cell" else _room(case["n"]), dtype=torch.float64, device=DEV)
    room[:len(areas)] = areas
    out = {"volumes": torch.cat([p[0] for p in parts]), "offsets": None, "neighbors": None, "areas": room}
    if kind == "cell":
        del out["offsets"]
    return out
