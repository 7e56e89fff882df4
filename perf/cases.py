"""Performance cases of slak_b200: what a program refining meshes with it does.

A program holds control meshes on the GPU and refines them, either through a
plan that is replayed whenever the positions move (``Plan``), through the
one-shot call of the scheme classes (``CatmullClark.subdivideIteratively``),
or many meshes at once (``Batch``).  The cases take each of these over both
schemes, closed and open meshes, triangles, quads and polygons, one level to
seven, and a thousand to sixty-five million refined quads.

A case is a dict of plain values:

    entry    "plan", "call" or "batch"
    scheme   "slak" or "lak"
    mesh     "torus", "tri", "mixed", "grid" or "cylinder" (not for a batch)
    w, h     the mesh's grid: w * h cells before merging and splitting
    levels   subdivision levels
    order    "grid": vertices and faces in grid order, "scattered": shuffled
    graph, autotune, compensated   plan / batch options
    creases  share of the edges that carry a crease (plans)
    count, fmin, fmax              a batch's meshes: how many, and their faces
    pick     seed of the topology; the seed of prepare() moves the vertices and
             renumbers them, so every case keeps its sizes
"""
import math
import random

import numpy as np
import torch

from slak_b200 import LAK, POLY, QUAD, SLAK, TRI, _abi, api

KINDS = ("torus", "tri", "mixed", "grid", "cylinder")


def listed():
    plan = {"entry": "plan", "order": "grid", "graph": True, "autotune": False, "compensated": False, "creases": 0.0, "pick": 1}
    call = dict(plan, entry="call", graph=False)
    batch = {"entry": "batch", "graph": True, "compensated": False, "pick": 2}
    return [
        # a small prop in a viewer, refined again on each frame: launches and latency
        dict(plan, name="torus32_slak_3", scheme="slak", mesh="torus", w=32, h=32, levels=3),
        # a small triangle model, the other scheme; the first level turns it into quads
        dict(plan, name="tri1280_lak_4", scheme="lak", mesh="tri", w=32, h=20, levels=4),
        # the large model of the benchmark: polygons of 3 to 8 sides, 65 million refined quads
        dict(plan, name="mixed512_slak_4", scheme="slak", mesh="mixed", w=512, h=512, levels=4, autotune=True),
        # the same with the other scheme, which also writes face offsets and corner positions
        dict(plan, name="mixed512_lak_4", scheme="lak", mesh="mixed", w=512, h=512, levels=4, autotune=True),
        # deep refinement of a model with two poles of valence 64, in the exact summation mode
        dict(plan, name="cylinder_slak_7", scheme="slak", mesh="cylinder", w=64, h=32, levels=7, compensated=True),
        # an open surface (cloth, terrain) with boundary rules, run without a graph
        dict(plan, name="grid300_slak_3", scheme="slak", mesh="grid", w=301, h=299, levels=3, graph=False),
        # a film model whose creases are live at the first levels
        dict(plan, name="creased_slak_3", scheme="slak", mesh="mixed", w=200, h=150, levels=3, creases=0.05),
        # one level of a large scan whose faces and vertices come in no order
        dict(plan, name="scan_lak_1", scheme="lak", mesh="tri", w=500, h=400, levels=1, order="scattered"),
        # the reference's own call in a modelling tool: a new mesh, refined once, results owned by the caller
        dict(call, name="call_mixed70_slak_2", scheme="slak", mesh="mixed", w=75, h=67, levels=2),
        # the same call on a quad model at export resolution
        dict(call, name="call_torus257_lak_3", scheme="lak", mesh="torus", w=257, h=255, levels=3),
        # a scene of small props, each with its own level of detail
        dict(batch, name="batch_small_slak", scheme="slak", count=32, fmin=100, fmax=2000),
        # a scene whose models differ in size by a factor of a thousand
        dict(batch, name="batch_uneven_slak", scheme="slak", count=32, fmin=100, fmax=100000),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    entry = rng.choice(("plan", "plan", "plan", "call", "batch"))
    case = {"entry": entry, "scheme": rng.choice(("slak", "lak")), "graph": entry != "call" and rng.random() < 0.7,
            "compensated": entry != "call" and rng.random() < 0.25, "pick": rng.randrange(1, 1 << 30)}
    if entry == "batch":
        fmin = _log_uniform(rng, 64, 1000)
        case.update(count=rng.randrange(2, 33), fmin=fmin, fmax=_log_uniform(rng, 2 * fmin, 60000))
        return case
    mesh = rng.choice(KINDS)
    faces = _log_uniform(rng, 64, 300000)
    h = max(5, int(round(math.sqrt(faces * rng.uniform(0.25, 1.0)))))
    w = max(5, faces // h)
    if mesh == "cylinder":
        w = rng.randrange(5, 97)
        h = max(2, min(faces, 60000) // w)
    levels = rng.randrange(1, 7)
    while levels > 1 and w * h * 6 * 4 ** (levels - 1) > 60_000_000:
        levels -= 1
    case.update(mesh=mesh, w=w, h=h, levels=levels, order=rng.choice(("grid", "grid", "scattered")),
                autotune=False, creases=rng.choice((0.0, 0.0, 0.03)) if entry == "plan" and mesh != "grid" else 0.0)
    return case


# ------------------------------------------------------------------ meshes
# A mesh's faces as a list of (k, order) blocks of vertex ids with a sort key
# per face; every mesh is manifold, with consistent orientation.

def _cells(w, h, closed):
    i, j = np.meshgrid(np.arange(w), np.arange(h), indexing="ij")
    i, j = i.ravel(), j.ravel()
    if closed:
        at = lambda a, b: (a % w) * h + b % h
    else:
        at = lambda a, b: a * (h + 1) + b
    return i, j, at


def _blocks(kind, w, h, rng):
    """(blocks of (key, ids), xyz) of the mesh."""
    if kind == "cylinder":                     # w segments, h rings of quads, a fan of triangles at each pole
        i, j = np.meshgrid(np.arange(h), np.arange(w), indexing="ij")
        i, j = i.ravel(), j.ravel()
        at = lambda a, b: a * w + b % w
        quads = np.stack([at(i, j), at(i, j + 1), at(i + 1, j + 1), at(i + 1, j)], 1)
        s, bottom, top = np.arange(w), (h + 1) * w, (h + 1) * w + 1
        low = np.stack([np.full(w, bottom), at(0, s + 1), at(0, s)], 1)
        high = np.stack([np.full(w, top), at(h, s), at(h, s + 1)], 1)
        n = h * w
        a, z = 2 * np.pi * np.tile(s, h + 1) / w, np.repeat(np.arange(h + 1) / h, w)
        xyz = np.concatenate([np.stack([np.cos(a), np.sin(a), 2 * z - 1], 1), [[0, 0, -1.0], [0, 0, 1.0]]])
        return [(np.arange(n), quads), (n + s, low), (n + w + s, high)], xyz
    i, j, at = _cells(w, h, kind != "grid")
    key = i * h + j
    quad = np.stack([at(i, j), at(i + 1, j), at(i + 1, j + 1), at(i, j + 1)], 1)
    if kind == "grid":
        a, b = np.meshgrid(np.arange(w + 1), np.arange(h + 1), indexing="ij")
        xyz = np.stack([a.ravel() / w, b.ravel() / h, np.zeros(a.size)], 1)
        return [(key, quad)], xyz
    a, b = np.meshgrid(2 * np.pi * np.arange(w) / w, 2 * np.pi * np.arange(h) / h, indexing="ij")
    a, b = a.ravel(), b.ravel()
    xyz = np.stack([(1 + 0.3 * np.cos(b)) * np.cos(a), (1 + 0.3 * np.cos(b)) * np.sin(a), 0.3 * np.sin(b)], 1)
    if kind == "torus":
        return [(key, quad)], xyz
    size = np.ones(w * h, dtype=np.int64)      # cells of the group that starts here, 0: part of the one before
    split = np.ones(w * h, dtype=bool)
    if kind == "mixed":                        # groups of two or three cells on every other row, single cells split
        u = rng.random_sample(w * h)
        start = (i % 2 == 0) & (i < w - w % 2) & (j % 3 == 0) & (j + 2 < h)
        m = np.where(start & (u < 0.12), 3, np.where(start & (u < 0.45), 2, 1))
        size = m.copy()
        for k in (1, 2):
            size[np.flatnonzero(m > k) + k] = 0
        split = (size == 1) & (rng.random_sample(w * h) < 0.03)
    out = [(2 * key[(size == 1) & ~split], quad[(size == 1) & ~split])]
    s = np.flatnonzero(split)
    q, d = quad[s], (rng.random_sample(s.size) < 0.5)[:, None]
    out.append((2 * key[s], np.where(d, q[:, [0, 1, 2]], q[:, [0, 1, 3]])))
    out.append((2 * key[s] + 1, np.where(d, q[:, [0, 2, 3]], q[:, [1, 2, 3]])))
    for m in (2, 3):
        s = np.flatnonzero(size == m)
        ids = [at(i[s], j[s])] + [at(i[s] + 1, j[s] + k) for k in range(m + 1)] + [at(i[s], j[s] + k) for k in range(m, 0, -1)]
        out.append((2 * key[s], np.stack(ids, 1)))
    return [(k, f) for k, f in out if k.size], xyz


def _topology(kind, w, h, pick):
    """(ptr, ids, xyz, type, largest face order) in grid order."""
    blocks, xyz = _blocks(kind, w, h, np.random.RandomState(pick % (1 << 32)))
    order = np.concatenate([np.full(k.size, f.shape[1]) for k, f in blocks])
    rank = np.empty(order.size, dtype=np.int64)
    by_key = np.argsort(np.concatenate([k for k, _ in blocks]), kind="stable")
    rank[by_key] = np.arange(order.size)
    ptr = np.concatenate([[0], np.cumsum(order[by_key])])
    ids = np.empty(ptr[-1], dtype=np.int64)
    at = 0
    for k, f in blocks:
        ids[(ptr[rank[at:at + k.size]][:, None] + np.arange(f.shape[1])).ravel()] = f.ravel()
        at += k.size
    lo, hi = int(order.min()), int(order.max())
    return ptr, ids, xyz, QUAD if lo == hi == 4 else TRI if lo == hi == 3 else POLY, hi


def _mesh(kind, w, h, pick, order, seed):
    """(ptr, ids, xyz, type, largest face order) as numpy arrays: positions and numbering from the seed."""
    ptr, ids, xyz, t, hi = _topology(kind, w, h, pick)
    rng = np.random.RandomState(seed % (1 << 32))
    nv = xyz.shape[0]
    if order == "scattered":
        new = rng.permutation(nv)
        faces = rng.permutation(ptr.size - 1)
        n = np.diff(ptr)[faces]
        to = np.concatenate([[0], np.cumsum(n)])
        ids = ids[np.repeat(ptr[faces] - to[:-1], n) + np.arange(ids.size)]
        ptr = to
    else:
        new = (np.arange(nv) + rng.randint(nv)) % nv
    moved = np.empty_like(xyz)
    moved[new] = xyz + rng.uniform(-0.002, 0.002, xyz.shape)
    return ptr.astype(np.int32), new[ids].astype(np.int32), moved.astype(np.float32), t, hi


def _device_mesh(ptr, ids, xyz, t, hi):
    n = np.diff(ptr)
    vals = (np.arange(ids.size) - np.repeat(ptr[:-1], n) + 1).astype(np.int32)
    pos = np.ones((xyz.shape[0], 4), dtype=np.float32)
    pos[:, :3] = xyz
    dev = [torch.from_numpy(a).cuda() for a in (ptr, ids, vals, pos.reshape(-1))]
    return api.DeviceMesh(t, n.size, xyz.shape[0], ids.size, hi, True, *dev)


def _creases(ptr, ids, share, seed):
    """Vertex pairs of some of the edges, each once, and their sharpness."""
    nxt = np.arange(1, ids.size + 1)
    nxt[ptr[1:] - 1] = ptr[:-1]
    a, b = ids, ids[nxt]
    rng = np.random.RandomState((seed + 7) % (1 << 32))
    up = np.flatnonzero(a < b)
    some = np.sort(rng.permutation(up)[:max(1, int(up.size * share))])
    return np.stack([a[some], b[some]], 1).astype(np.int32), rng.choice([0.5, 1.0, 2.0, 3.0], some.size).astype(np.float32)


def _items(case):
    """A batch's meshes: (kind, w, h, levels, pick) of each."""
    rng = random.Random(case["pick"])
    out = []
    for _ in range(case["count"]):
        faces = _log_uniform(rng, case["fmin"], case["fmax"])
        kind = rng.choice(("torus", "torus", "tri", "mixed"))
        h = max(5, int(round(math.sqrt(faces / rng.uniform(1.0, 4.0)))))
        out.append((kind, max(6, faces // h // (2 if kind == "tri" else 1)), h, rng.randrange(1, 5), rng.randrange(1 << 30)))
    return out


# ------------------------------------------------------------------ the path
def _scheme(case):
    return LAK if case["scheme"] == "lak" else SLAK


def _flags(case):
    return ((_abi.PLAN_GRAPH if case["graph"] else 0) | (_abi.PLAN_AUTOTUNE if case.get("autotune") else 0)
            | (_abi.PLAN_COMPENSATED if case["compensated"] else 0))


class _Kept(dict):
    """Arrays of refined meshes; they live as long as their owner (mesh, plan or batch)."""

    def __init__(self, arrays, owner):
        super().__init__(arrays)
        self.owner = owner


def _arrays(m):
    out = {"ids": m.ids, "verts": m.verts}
    if m.ptr is not None:
        out.update(ptr=m.ptr, vals=m.vals)
    return out


def prepare(case, seed):
    if case["entry"] == "batch":
        items = _items(case)
        meshes = [_device_mesh(*_mesh(kind, w, h, pick, "grid", seed + 31 * k)) for k, (kind, w, h, _, pick) in enumerate(items)]
        batch = api.Batch(meshes, [it[3] for it in items], _scheme(case), _flags(case))
        out = {str(k): [m.ids, m.verts] for k, m in enumerate(batch.output(k) for k in range(len(items)))}
        return {"plan": batch, "stream": _stream(case), "out": _Kept(out, batch)}
    host = _mesh(case["mesh"], case["w"], case["h"], case["pick"], case["order"], seed)
    mesh = _device_mesh(*host)
    if case["entry"] == "call":
        return {"mesh": mesh, "levels": case["levels"], "scheme": api.LAKCatmullClark if case["scheme"] == "lak" else api.CatmullClark}
    creases = _creases(host[0], host[1], case["creases"], seed) if case["creases"] else None
    plan = api.Plan(mesh, case["levels"], _scheme(case), _flags(case), creases=creases)
    return {"plan": plan, "stream": _stream(case), "out": _Kept(_arrays(plan.output()), plan)}


_OWN = []


def _stream(case):
    """A graph is captured and replayed on the program's own stream (one for all its plans)."""
    if not case["graph"]:
        return None
    if not _OWN:
        _OWN.append(torch.cuda.Stream())
    _OWN[0].wait_stream(torch.cuda.current_stream())
    return _OWN[0]


def run(state):
    if "plan" in state:
        state["plan"].execute(state["stream"])
        return state["out"]
    refined = api.DeviceMesh()
    state["scheme"].subdivideIteratively(state["mesh"], refined, state["levels"])
    return _Kept(_arrays(refined), refined)


# ------------------------------------------------------------------ sizes
def _sizes(kind, w, h, pick, levels, lak):
    """Compulsory bytes and operations: the control mesh in, the refined mesh out; every level's positions."""
    ptr, ids, xyz, t, _ = _topology(kind, w, h, pick)
    f, n, v, b = ptr.size - 1, ids.size, xyz.shape[0], 2 * (w + h) if kind == "grid" else 0
    total, flops = 4 * n + 16 * v + (0 if t == QUAD else 4 * (f + 1)), 0
    for _ in range(levels):
        e = (n - b) // 2 + b
        v, f, n, b = v + f + e, n, 4 * n, 2 * b
        flops += 4 * 10 * v
    return total + 4 * n + 16 * v + (4 * n + 4 * (f + 1) if lak else 0), flops


def work(case):
    lak = case["scheme"] == "lak"
    if case["entry"] == "batch":
        got = [_sizes(kind, w, h, pick, levels, lak) for kind, w, h, levels, pick in _items(case)]
    else:
        got = [_sizes(case["mesh"], case["w"], case["h"], case["pick"], case["levels"], lak)]
    return {"bytes": sum(g[0] for g in got), "flops": sum(g[1] for g in got)}


# ------------------------------------------------------------------ 64 bits
def exact(case, seed):
    lak = case["scheme"] == "lak"
    if case["entry"] == "batch":
        return {str(k): [None, _refine(*_mesh(kind, w, h, pick, "grid", seed + 31 * k)[:3], levels, lak)]
                for k, (kind, w, h, levels, pick) in enumerate(_items(case))}
    ptr, ids, xyz = _mesh(case["mesh"], case["w"], case["h"], case["pick"], case["order"], seed)[:3]
    creases = _creases(ptr, ids, case["creases"], seed) if case["creases"] else None
    out = {"ids": None, "verts": _refine(ptr, ids, xyz, case["levels"], lak, creases)}
    if lak:
        out.update(ptr=None, vals=None)
    return out


def _refine(ptr, ids, xyz, levels, lak, creases=None):
    """Catmull-Clark positions in float64 with the schemes' vertex numbering:
    [old vertices | face points | edge points], quad c of a refined mesh from
    corner c, edges numbered by (tail, corner) of their owning half-edge (the
    lower id's, or a boundary edge's only one) or, LAK, by (higher, lower) end."""
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    pos = torch.ones(xyz.shape[0], 4, dtype=torch.float64)
    pos[:, :3] = torch.from_numpy(xyz).double()
    pos, ids = pos.to(dev), torch.from_numpy(ids).long().to(dev)
    ptr = torch.from_numpy(ptr).long().to(dev)
    n = ids.numel()
    c = torch.arange(n, device=dev)
    face = torch.repeat_interleave(torch.arange(ptr.numel() - 1, device=dev), ptr.diff())
    nxt, prv = c + 1, c - 1
    nxt[ptr[1:] - 1] = ptr[:-1]
    prv[ptr[:-1]] = ptr[1:] - 1
    nf = ptr.numel() - 1
    sharp = None                                # per corner: sharpness of its half-edge's edge
    if creases is not None:
        nv = pos.shape[0]
        key = torch.minimum(ids, ids[nxt]) * nv + torch.maximum(ids, ids[nxt])
        pairs, s = (torch.from_numpy(x).to(dev) for x in creases)
        want, at = (pairs.long().amin(1) * nv + pairs.long().amax(1)).sort()
        hit = torch.searchsorted(want, key).clamp(max=want.numel() - 1)
        sharp = torch.where(want[hit] == key, s.double()[at][hit], 0.0)
    for level in range(levels):
        if level:                               # a refined level: quads
            n = ids.numel()
            nf = n // 4
            c = torch.arange(n, device=dev)
            face, nxt, prv = c // 4, (c & ~3) | ((c + 1) & 3), (c & ~3) | ((c + 3) & 3)
        nv = pos.shape[0]
        head = ids[nxt]
        lo, hi = torch.minimum(ids, head), torch.maximum(ids, head)
        keys, edge, seen = torch.unique(hi * nv + lo, return_inverse=True, return_counts=True)
        ne = keys.numel()
        if not lak:
            own = torch.nonzero((ids < head) | (seen[edge] == 1)).flatten()
            own = own[torch.sort(ids[own], stable=True).indices]
            number = torch.empty(ne, dtype=torch.long, device=dev)
            number[edge[own]] = torch.arange(ne, device=dev)
            edge = number[edge]
            seen = torch.bincount(edge, minlength=ne)
        del keys, lo, hi
        add = lambda size, index, what: torch.zeros(size, 4, dtype=torch.float64, device=dev).index_add_(0, index, what)
        count = lambda index, size: torch.bincount(index, minlength=size).double()[:, None]
        fp = add(nf, face, pos[ids]) / count(face, nf)
        single = (seen == 1)[:, None]
        mid = add(ne, edge, pos[ids] + pos[head]) / (2 * seen[:, None])
        ep = torch.where(single, mid, mid / 2 + add(ne, edge, fp[face]) / 4)
        valence = count(ids, nv)
        vp = (add(nv, ids, pos[head]) + add(nv, ids, fp[face])) / valence ** 2 + pos * (valence - 2) / valence
        rim = torch.nonzero(seen[edge] == 1).flatten()
        if rim.numel():
            a, b = ids[rim], head[rim]
            vp[a] = 0.75 * pos[a]
            vp.index_add_(0, a, pos[b] / 8).index_add_(0, b, pos[a] / 8)
        if sharp is not None:
            s = torch.zeros(ne, dtype=torch.float64, device=dev)
            s[edge] = sharp
            w = s.clamp(max=1.0)[:, None]
            ep = ep * (1 - w) + mid * w
            live = torch.nonzero((sharp > 0) & (ids < head)).flatten()     # each crease edge once
            a, b = ids[live], head[live]
            k = torch.bincount(torch.cat([a, b]), minlength=nv)
            total = torch.zeros(nv, dtype=torch.float64, device=dev)
            total.index_add_(0, a, sharp[live]).index_add_(0, b, sharp[live])
            ends = torch.zeros_like(pos).index_add_(0, a, pos[b]).index_add_(0, b, pos[a])
            rule = torch.where((k == 2)[:, None], 0.75 * pos + ends / 8, pos)
            w = torch.where(k >= 2, (total / k.clamp(min=1)).clamp(max=1.0), 0.0)[:, None]
            vp = vp * (1 - w) + rule * w
            s = (sharp - 1).clamp(min=0)
            sharp = torch.stack([s, torch.zeros_like(s), torch.zeros_like(s), s[prv]], 1).flatten()
        ids = torch.stack([ids, nv + nf + edge, nv + face, nv + nf + edge[prv]], 1).flatten() if level + 1 < levels else None
        pos = torch.cat([vp, fp, ep])
    return pos.flatten()
