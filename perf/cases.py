"""The work that users of this library have it do, as cases to be timed: one plain
query, batches of queries, tree builds, interval scans, metacell formation, marching
cubes and the whole isosurface path, each through the package's public calls, from the
smallest calls (where latency and launches count) to the 2^28-point batch.

The library leaves the order of a query's results unspecified (as the reference's GPU
searches do), and a caller takes them as they come.  Answer therefore holds the result
buffers as the call left them, and puts a query's records in ascending order, all of
them, when somebody reads them to compare; what has no fixed length is then followed by
zeros up to the most the case allows for.  Likewise a built tree is copied to the host
only when it is read."""
import importlib
import math

import numpy as np
import torch

pst = importlib.import_module("static-priority-search-tree_b200")

DOMAIN, SPREAD = float(1 << 24), float(1 << 16)  # "uniform" points: dim1 ~ U[0, 2^24), dim2 - dim1 ~ U[0, 2^16)
GAP = 0.01                                       # "gaps" points: dim1 ~ U[0, 1), dim2 - dim1 ~ Exp(0.01)
KINDS = {"three": 0, "left": 1, "right": 2}
VALUE = {"f32": torch.float32, "f64": torch.float64, "i32": torch.int32}


def listed():
    return [
        # one isovalue over the metacells of a small volume: a single small call, all latency
        {"name": "query-isovalue-65k", "op": "query", "data": "volume", "px": 257, "py": 253, "pz": 65, "mc": 4,
         "dt": "f32", "ids": "indices", "ret": "ids", "kind": "left", "sel": 0.0},
        # one 3-sided range query on a large tree, as a program that answers one user at a time calls it
        {"name": "query-three-67m", "op": "query", "data": "uniform", "n": 1 << 26, "dt": "f32", "ids": "indices",
         "ret": "ids", "kind": "three", "sel": 1e-3},
        # a sweep over 16 isovalues of the 512^3 volume's metacells: a small batch on an ordinary tree
        {"name": "batch-16-isovalues-2m", "op": "batch", "data": "volume", "px": 512, "py": 512, "pz": 512, "mc": 4,
         "dt": "f32", "ids": "indices", "ret": "ids", "nq": 16, "sync": True},
        # doubles with whole points returned, odd sizes
        {"name": "batch-601-points-f64", "op": "batch", "data": "uniform", "n": 12_345_677, "dt": "f64",
         "ids": "indices", "ret": "points", "nq": 601, "sync": True},
        # the headline: 4096 mixed queries over 2^28 points, queries and results on the device
        {"name": "batch-4096-mixed-268m", "op": "batch", "data": "uniform", "n": 1 << 28, "dt": "f32",
         "ids": "indices", "ret": "ids", "nq": 4096, "sync": False},
        # the tree of the 512^3 volume's metacells, rebuilt for each volume of a time series
        {"name": "build-metacells-2m", "op": "build", "data": "volume", "px": 512, "py": 512, "pz": 512, "mc": 4,
         "dt": "f32", "ids": "indices"},
        # doubles whose ids come in no order (records gathered from elsewhere), an odd count
        {"name": "build-5m-f64-shuffled", "op": "build", "data": "uniform", "n": 5_000_011, "dt": "f64",
         "ids": "shuffled"},
        # a large tree
        {"name": "build-67m", "op": "build", "data": "uniform", "n": 1 << 26, "dt": "f32", "ids": "indices"},
        # the interval scan a user runs where there is no tree, over more than L2 holds
        {"name": "scan-134m", "op": "scan", "data": "uniform", "n": (1 << 27) - 77, "dt": "f32", "ids": "indices",
         "ret": "ids"},
        # metacells of a volume whose rows are not a multiple of four vertices
        {"name": "metacells-odd", "op": "metacells", "px": 509, "py": 381, "pz": 263, "mc": 4, "dt": "f32",
         "ids": "indices"},
        # triangles of one isovalue's active metacells, in the order a query gave them (none in space)
        {"name": "triangles-512", "op": "triangles", "px": 512, "py": 512, "pz": 512, "mc": 4, "iso": 0.23},
        # the whole isosurface path: volume -> metacells -> tree -> query -> triangles
        {"name": "isosurface-384", "op": "isosurface", "px": 384, "py": 384, "pz": 384, "mc": 4, "iso": 0.17},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | rng.randint(0, 1)

    def volume(lo, hi):
        return {"px": size(lo, hi), "py": size(lo, hi), "pz": size(lo, hi)}

    op = rng.choice(["query", "query", "batch", "batch", "build", "build", "scan", "metacells", "triangles",
                     "isosurface"])
    dt = rng.choice(["f32", "f32", "f64", "i32"])
    ids = rng.choice(["indices", "indices", "shuffled", "none"])
    ret = "points" if ids == "none" else rng.choice(["ids", "ids", "points"])
    if op == "query":
        return {"op": op, "data": "uniform", "n": size(1 << 14, 1 << 26), "dt": dt, "ids": ids, "ret": ret,
                "kind": rng.choice(["three", "left", "right"]), "sel": math.exp(rng.uniform(math.log(1e-5), math.log(1e-1)))}
    if op == "batch":
        data = "gaps" if dt == "f32" and rng.random() < 0.5 else "uniform"
        return {"op": op, "data": data, "n": size(1 << 16, 1 << 26), "dt": dt, "ids": ids, "ret": ret,
                "nq": size(2, 4096), "sync": rng.random() < 0.5}
    if op == "build":
        return {"op": op, "data": "uniform", "n": size(1 << 14, 1 << 26), "dt": dt, "ids": ids}
    if op == "scan":
        return {"op": op, "data": "uniform", "n": size(1 << 18, 1 << 27), "dt": dt, "ids": ids, "ret": ret}
    if op == "metacells":
        return {"op": op, **volume(96, 512), "mc": rng.choice([1, 2, 4, 4, 8]), "dt": dt, "ids": rng.choice(["indices", "none"])}
    iso = round(rng.uniform(0.1, 0.8), 3)
    return {"op": op, **volume(96, 512 if op == "triangles" else 384), "mc": rng.choice([2, 4, 4, 8]), "iso": iso}


# ---------------------------------------------------------------------------
# inputs


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _volume(c, seed):
    """32 Gaussian blobs (sigma 8..40 voxels) and a little noise, (pz, py, px); integers for i32."""
    rng = np.random.default_rng(seed)
    dims = [c["px"], c["py"], c["pz"]]
    vol = torch.zeros(dims[::-1], dtype=torch.float32, device="cuda")
    for _ in range(32):
        mid, s, a = rng.uniform([0, 0, 0], dims), rng.uniform(8.0, 40.0), float(rng.uniform(0.5, 1.0))
        lo = [max(int(m - 4 * s), 0) for m in mid]
        hi = [min(int(m + 4 * s) + 2, d) for m, d in zip(mid, dims)]
        gx, gy, gz = [torch.exp(-0.5 * ((torch.arange(l, h, device="cuda", dtype=torch.float32) - float(m)) / s) ** 2)
                      for l, h, m in zip(lo, hi, mid)]
        vol[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]] += a * gz[:, None, None] * gy[None, :, None] * gx
    vol += 0.01 * torch.randn(vol.shape, generator=_gen(seed), device="cuda")
    if c.get("dt", "f32") == "i32":
        vol = (vol * 4096).to(torch.int32)
    return vol.to(VALUE[c.get("dt", "f32")])


def _points(c, seed):
    """PointStruct records on the device: one row of 4- or 8-byte words a point."""
    if c["data"] == "volume":
        dims = [c["px"], c["py"], c["pz"]]
        rec, n = pst.formMetacellTags(_volume(c, seed), dims, [c["mc"]] * 3, c["dt"], c["ids"] != "none")
        return rec.view(torch.int32).view(n, -1)
    n, t, g = c["n"], VALUE[c["dt"]], _gen(seed)
    word = torch.int64 if c["dt"] == "f64" else torch.int32
    rec = torch.empty((n, 2 if c["ids"] == "none" else 3), dtype=word, device="cuda")
    if c["dt"] == "i32":
        d1 = torch.randint(0, int(DOMAIN), (n,), generator=g, device="cuda", dtype=t)
        d2 = d1 + torch.randint(0, int(SPREAD), (n,), generator=g, device="cuda", dtype=t)
    elif c["data"] == "gaps":
        d1 = torch.rand(n, generator=g, device="cuda", dtype=t)
        d2 = d1 + torch.empty(n, device="cuda", dtype=t).exponential_(1.0 / GAP, generator=g)
    else:
        d1 = torch.rand(n, generator=g, device="cuda", dtype=t) * DOMAIN
        d2 = d1 + torch.rand(n, generator=g, device="cuda", dtype=t) * SPREAD
    rec[:, 0], rec[:, 1] = d1.view(word), d2.view(word)
    if c["ids"] == "shuffled":
        rec[:, 2] = torch.randperm(n, generator=g, device="cuda", dtype=torch.int64).to(word)
    elif c["ids"] == "indices":
        rec[:, 2] = torch.arange(n, device="cuda", dtype=word)
    return rec


def _bounds(c, kinds, sel, anchor):
    """Bounds (min1, max1, min2) that about a share `sel` of the points meets; anchor in [0, 1)."""
    gaps = c["data"] == "gaps"
    dom, w = (1.0, 0.0) if gaps else (DOMAIN, SPREAD)
    a = anchor * dom * (1 - np.minimum(2 * sel, 0.9))

    def below(share):  # dim2 bound, from the dim1 bound b down, that a share of the points with dim1 <= b meets
        if gaps:
            return np.where(share < GAP, -GAP * np.log(share / GAP), GAP - share)
        return np.where(share < w / (2 * dom), w - np.sqrt(2 * w * dom * share), w / 2 - share * dom)

    three, left = kinds == 0, kinds == 1
    b = np.maximum(a, dom * sel + w)
    min1 = np.where(three, a, np.where(left, 0.0, a * (1 - np.minimum(sel + 0.01, 0.9))))
    max1 = np.where(three, a + sel * dom, np.where(left, b, 0.0))
    min2 = np.where(three, a, np.where(left, b + below(sel), dom + below(sel)))
    return min1, max1, min2


def _queries(c, seed, nq):
    rng = np.random.default_rng(seed)
    if c["data"] == "volume":  # isovalues above the noise, over most of the blobs' range
        iso = rng.uniform(0.06, 0.95, nq)
        return pst.make_queries([KINDS["left"]] * nq, iso * 0, iso, iso, c["dt"])
    if c["op"] == "query":
        kinds, sel = np.full(nq, KINDS[c["kind"]]), np.full(nq, c["sel"])
    else:  # half 3-sided, a quarter each 2-sided, selectivities log-uniform over [1e-7, 1e-2]
        kinds = rng.permutation(np.repeat([0, 1, 2], [nq - 2 * (nq // 4), nq // 4, nq // 4]))
        sel = np.exp(rng.uniform(math.log(1e-7), math.log(1e-2), nq))
    return pst.make_queries(kinds, *_bounds(c, kinds, sel, rng.random(nq)), c["dt"])


def _value(c, word):
    """A query's bound as the plain number that the single-query calls take."""
    return np.array([word], np.uint64).view({"f32": np.float32, "f64": np.float64, "i32": np.int32}[c["dt"]])[0].item()


def _metacells(c):
    return math.prod(-(-(c[p] - 1) // c["mc"]) for p in ("px", "py", "pz"))


def _room(c):
    """Records (or triangles) that a case's results may come to: the room a caller gives them."""
    if c["op"] in ("triangles", "isosurface"):
        return _metacells(c) * c["mc"] ** 3 // 4 + 1024
    if "n" not in c:
        return _metacells(c) * c.get("nq", 1)
    if c["op"] == "scan":
        return c["n"] // 128 + 1024
    if c["op"] == "query":
        return min(c["n"], int(2 * c["sel"] * c["n"]) + 4096)
    share = min(c["nq"] * 1e-2, c["nq"] * 8.7e-4 + 6 * 0.0019 * c["nq"] ** 0.5)  # the mean and six deviations
    return int(1.02 * share * c["n"]) + 64 * c["nq"] + 4096


def _record_bytes(c):
    return pst.point_dtype(c["dt"], c["ids"] != "none").itemsize


def prepare(case, seed):
    c = case
    if c["op"] in ("query", "batch"):
        pts = _points(c, seed)
        n, size = len(pts), 4 if c["ret"] == "ids" else _record_bytes(c)
        tree = pst.StaticPSTGPU(pts, n, c["dt"], c["ids"] != "none")
        del pts
        if c["op"] == "query":
            q = _queries(c, seed, 1)[0]
            return {"case": c, "tree": tree, "bounds": [_value(c, q[f]) for f in ("min1", "max1", "min2")],
                    "out": torch.empty(_room(c) * size, dtype=torch.uint8, device="cuda")}
        q = _queries(c, seed, c["nq"])
        engine = pst.BatchEngine(tree, c["nq"])
        engine.count(q)  # a caller looks at the counts once, before it gives the results a buffer
        if not c["sync"]:
            q = torch.from_numpy(q.view(np.uint8).copy()).cuda()
        return {"case": c, "tree": tree, "engine": engine, "queries": q,
                "out": torch.empty(_room(c) * size, dtype=torch.uint8, device="cuda"),
                "offsets": torch.empty(c["nq"] + 1, dtype=torch.int64, device="cuda")}
    if c["op"] == "build":
        return {"case": c, "points": _points(c, seed)}
    if c["op"] == "scan":
        v = float(np.random.default_rng(seed).uniform(0.1, 0.9)) * DOMAIN
        return {"case": c, "points": _points(c, seed), "value": int(v) if c["dt"] == "i32" else v}
    state = {"case": c, "volume": _volume(c, seed), "dims": [c["px"], c["py"], c["pz"]], "mc": [c["mc"]] * 3}
    if c["op"] == "triangles":
        active = _active(c, state["volume"])
        state["ids"] = active[torch.randperm(len(active), generator=_gen(seed), device="cuda")].to(torch.int32)
    elif c["op"] == "isosurface":
        n = pst.calcNumMetacells(state["dims"], state["mc"])[1]
        state["ids"] = torch.empty(n, dtype=torch.int32, device="cuda")
    return state


# ---------------------------------------------------------------------------
# one pass


def run(state):
    c = state["case"]
    if c["op"] == "query":
        min1, max1, min2 = state["bounds"]
        n = state["tree"].search_into(c["kind"], state["out"], _room(c), min1, max1, min2, ret=c["ret"])
        return Answer(count=n, records=lambda: _ascending(c, state["out"], [0, n]))
    if c["op"] == "batch":
        state["engine"].run(state["queries"], state["out"], state["offsets"], ret=c["ret"],
                            queries_on_device=not c["sync"], sync=c["sync"])
        return Answer(offsets=state["offsets"],
                      records=lambda: _ascending(c, state["out"], state["offsets"].tolist()))
    if c["op"] == "build":
        tree = pst.StaticPSTGPU(state["points"], len(state["points"]), c["dt"], c["ids"] != "none")
        return Answer({k: (lambda k=k: _exported(tree, k)) for k in ("dim1", "dim2", "med", "ids", "bitcodes")})
    if c["op"] == "scan":
        found = pst.intervalParallelSearch(state["points"], len(state["points"]), state["value"], c["dt"],
                                           c["ids"] != "none", c["ret"])
        return Answer(count=len(found),
                      records=lambda: _ascending(c, torch.from_numpy(found.view(np.uint8)).cuda(), [0, len(found)]))
    if c["op"] == "metacells":
        rec, n = pst.formMetacellTags(state["volume"], state["dims"], state["mc"], c["dt"], c["ids"] != "none")
        return Answer(records=lambda: _words(c, rec, n))
    if c["op"] == "triangles":
        tri = pst.marchingCubes(state["volume"], state["dims"], state["mc"], state["ids"], c["iso"])
        return Answer(count=len(tri), triangles=lambda: _padded(tri, _room(c)))
    rec, n = pst.formMetacellTags(state["volume"], state["dims"], state["mc"])
    tree = pst.StaticPSTGPU(rec, n)
    found = tree.search_into("left", state["ids"], n, max1=c["iso"], min2=c["iso"])
    tree.close()
    ids = state["ids"][:found].sort().values  # neighbours in the volume next to one another
    tri = pst.marchingCubes(state["volume"], state["dims"], state["mc"], ids, c["iso"])
    return Answer(count=found, ids=lambda: _padded(ids, n), triangles=lambda: _padded(tri, _room(c)))


class Answer(dict):
    """What a call left, by name; an entry that is a function makes its value when it is read."""

    def __getitem__(self, key):
        v = super().__getitem__(key)
        return v() if callable(v) else v


def _padded(rows, n):
    """The rows, then zeros up to n of them."""
    out = torch.zeros((n, *rows.shape[1:]), dtype=rows.dtype, device="cuda")
    out[:len(rows)] = rows
    return out


def _words(c, raw, n):
    """n records as rows of 32-bit words, without a record's padding."""
    size = 4 if c.get("ret") == "ids" else _record_bytes(c)
    words = raw[: n * size].view(torch.int32).view(n, size // 4)
    return words[:, :5] if size == 24 else words


def _ascending(c, raw, offsets):
    """All records, each query's in ascending order (by id, or by their words where they have none)."""
    rows, q = _words(c, raw, offsets[-1]), 0
    out = torch.zeros((_room(c), rows.shape[1]), dtype=torch.int32, device="cuda")
    while q + 1 < len(offsets):  # some queries at a time, about 2^26 records
        e = q + 1
        while e + 1 < len(offsets) and offsets[e + 1] - offsets[q] <= 1 << 26:
            e += 1
        part = rows[offsets[q]:offsets[e]]
        order = None
        for w in ([part.shape[1] - 1] if c["ids"] != "none" else range(part.shape[1])):
            key = part[:, w] if order is None else part[order, w]
            by = key.sort(stable=True).indices
            order = by if order is None else order[by]
        sizes = torch.tensor(offsets[q:e + 1], device="cuda").diff()
        query = torch.repeat_interleave(torch.arange(e - q, dtype=torch.int32, device="cuda"), sizes)
        order = order[query[order].sort(stable=True).indices]
        out[offsets[q]:offsets[e]] = part[order]
        q = e
    return out


def _exported(tree, name):
    """One field of the built tree in the reference's layout; values as their bits."""
    v = tree.export()[name]
    return np.zeros(0, np.int32) if v is None else v if v.itemsize == 1 else v.view(f"i{v.itemsize}")


# ---------------------------------------------------------------------------
# what a pass cannot do without


def work(case):
    c = case
    n = c["n"] if "n" in c else _metacells(c)
    if c["op"] in ("triangles", "isosurface"):
        # about 5 % of the cells' metacells are active, with close to one triangle a cell:
        # the vertices of the active metacells read, nine floats a triangle written
        cells = 0.05 * n * c["mc"] ** 3
        need = 4 * cells + 36 * cells
        return {"bytes": need if c["op"] == "triangles" else need + 4 * c["px"] * c["py"] * c["pz"], "flops": 27 * cells}
    size = _record_bytes(c)
    value = 8 if c["dt"] == "f64" else 4
    if c["op"] == "metacells":
        return {"bytes": value * c["px"] * c["py"] * c["pz"] + size * n, "flops": 0}
    if c["op"] == "build":  # every point read, every node (two values, the median of half of them, the id) written
        return {"bytes": n * (2 * size + value / 2), "flops": 0}
    back = 4 if c["ret"] == "ids" else size
    if c["op"] == "scan":  # the points read, one in 512 reported
        hits = n * SPREAD / 2 / DOMAIN
        return {"bytes": n * size + hits * back, "flops": 0}
    if c["op"] == "query":
        hits = n * (c["sel"] or 0.05)
        return {"bytes": max(hits, 1) * (value + 2 * back), "flops": 0}
    mean = 0.05 if c["data"] == "volume" else (1e-2 - 1e-7) / math.log(1e5)
    hits = c["nq"] * mean * n
    return {"bytes": min(hits, n) * (value + back) + hits * back + 32 * c["nq"], "flops": 0}


# ---------------------------------------------------------------------------
# 64-bit results


def _active(c, vol):
    """Ids of the metacells whose values span the isovalue, ascending."""
    lo, hi = vol, vol
    for axis in (2, 1, 0):
        size, mc = vol.shape[axis], c["mc"]
        cells = size - 1
        at = torch.arange(-(-cells // mc) * mc, device="cuda").clamp(max=cells)
        at = torch.cat([at.view(-1, mc), (at.view(-1, mc)[:, -1:] + 1).clamp(max=cells)], 1)
        shape = list(lo.shape)
        shape[axis:axis + 1] = list(at.shape)
        lo = lo.index_select(axis, at.reshape(-1)).view(shape).amin(axis + 1)
        hi = hi.index_select(axis, at.reshape(-1)).view(shape).amax(axis + 1)
    iso = torch.tensor(c["iso"], dtype=torch.float32, device="cuda")
    return ((lo <= iso) & (iso <= hi)).view(-1).nonzero().view(-1)


def _corner(axis, u, v):
    """Lower corner (bits x, y, z) of the cell edge along `axis` at the other two coordinates (u, v)."""
    other = [a for a in range(3) if a != axis]
    return (u << other[0]) | (v << other[1])


def _table():
    """Triangles of the 256 inside patterns as edge triples (edge 4 axis + u + 2 v): on a face with four
    crossings each inside corner is cut off by itself; loops are turned so that their normal points from
    inside to outside, begin at their smallest edge and are fanned from the first vertex whose diagonals
    leave the faces of the cube."""
    ends = [(_corner(a, u, v), _corner(a, u, v) | (1 << a)) for a in range(3) for v in range(2) for u in range(2)]
    number = {frozenset(e): i for i, e in enumerate(ends)}
    rings = []
    for a in range(3):
        p, q = [x for x in range(3) if x != a]
        rings += [[(s << a) | (i << p) | (j << q) for i, j in ((0, 0), (1, 0), (1, 1), (0, 1))] for s in range(2)]
    faces = [{f for f, r in enumerate(rings) if set(e) <= set(r)} for e in ends]
    spot = np.array([[(x >> d) & 1 for d in range(3)] for x in range(8)])
    table = []
    for inside in range(256):
        into = lambda x: (inside >> x) & 1  # noqa: E731
        near = {}
        for ring in rings:
            edge = [number[frozenset((ring[i], ring[(i + 1) % 4]))] for i in range(4)]
            cut = [i for i in range(4) if into(ring[i]) != into(ring[(i + 1) % 4])]
            pairs = [(edge[cut[0]], edge[cut[1]])] if len(cut) == 2 else [
                (edge[i - 1], edge[i]) for i in range(4) if into(ring[i])] if len(cut) == 4 else []
            for x, y in pairs:
                near.setdefault(x, []).append(y)
                near.setdefault(y, []).append(x)
        triangles, seen = [], set()
        for first in sorted(near):
            if first in seen:
                continue
            loop, step = [first], min(near[first])
            while step != first:
                loop.append(step)
                step = [x for x in near[step] if x != loop[-2]][0] if near[step][0] == loop[-2] else near[step][0]
            seen.update(loop)
            mids = np.array([spot[ends[e][0]] + spot[ends[e][1]] for e in loop])
            normal = np.cross(mids, np.roll(mids, -1, 0)).sum(0)
            outward = sum((spot[b] - spot[a]) if into(a) else (spot[a] - spot[b]) for a, b in (ends[e] for e in loop))
            if normal @ outward < 0:
                loop.reverse()
            k = loop.index(min(loop))
            loop = loop[k:] + loop[:k]
            m = len(loop)
            apex = next(j for j in range(m) if all(not faces[loop[j]] & faces[loop[(j + i) % m]] for i in range(2, m - 1)))
            triangles += [[loop[apex], loop[(apex + i) % m], loop[(apex + i + 1) % m]] for i in range(1, m - 1)]
        table.append(triangles)
    return ends, table


def _triangles64(c, vol, ids):
    """The triangles of the given metacells, in their order, in 64 bits."""
    ends, table = _table()
    most = max(map(len, table))
    count = torch.tensor([len(t) for t in table], device="cuda")
    edges = torch.tensor([t + [[0, 0, 0]] * (most - len(t)) for t in table], device="cuda")
    mc, dims = c["mc"], [c["px"], c["py"], c["pz"]]
    grid = [-(-(d - 1) // mc) for d in dims]
    cell = torch.arange(mc ** 3, device="cuda")
    at = torch.stack([ids % grid[0], ids // grid[0] % grid[1], ids // (grid[0] * grid[1])], 1)[:, None] * mc
    at = (at + torch.stack([cell % mc, cell // mc % mc, cell // mc ** 2], 1)).view(-1, 3)
    at = at[(at < torch.tensor(dims, device="cuda") - 1).all(1)]
    flat = vol.reshape(-1)
    corner = at[:, 0] + dims[0] * (at[:, 1] + dims[1] * at[:, 2])
    step = [(x & 1) + dims[0] * ((x >> 1 & 1) + dims[1] * (x >> 2)) for x in range(8)]
    iso = torch.tensor(c["iso"], dtype=torch.float32, device="cuda")
    inside = sum((flat[corner + s] >= iso).long() << x for x, s in enumerate(step))
    of = torch.repeat_interleave(torch.arange(len(at), device="cuda"), count[inside])
    nth = torch.arange(len(of), device="cuda") - (count[inside].cumsum(0) - count[inside])[of]
    low = torch.tensor([e[0] for e in ends], device="cuda")
    steps = torch.tensor(step, device="cuda")
    out = torch.empty((len(of), 3, 3), dtype=torch.float64, device="cuda")
    for v in range(3):
        edge = edges[inside[of], nth, v]
        axis, a = edge // 4, low[edge]
        fa = flat[corner[of] + steps[a]].double()
        fb = flat[corner[of] + steps[a | (1 << axis)]].double()
        t = (iso.double() - fa) / (fb - fa)
        for d in range(3):
            out[:, v, d] = at[of, d] + (a >> d & 1) + torch.where(axis == d, t, 0.0)
    return out.view(-1, 9)


def exact(case, seed):
    if case["op"] not in ("triangles", "isosurface"):
        return None  # ids, copied values and the order of a tree: compared as they are
    c, vol = case, _volume(case, seed)
    ids = _active(c, vol)
    if c["op"] == "triangles":
        ids = ids[torch.randperm(len(ids), generator=_gen(seed), device="cuda")]
    return {"triangles": _padded(_triangles64(c, vol, ids), _room(c))}
