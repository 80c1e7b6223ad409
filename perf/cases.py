"""Performance cases of the mesh spatial joins.

Each case is a call that a user of the library makes on datasets it has in
hand: joins of two resident datasets (overlap, intersection, containment;
hash, two-pass and learned sizing; exact and float32 predicates), a batch of
small joins replayed as one captured graph, and whole queries that start from
host arrays, as the command-line tools and services run them.  Meshes are the
library's own generated workloads; sizes run from a handful of meshes to
hundreds of thousands.

A pass ends with the pairs in the caller's own pinned buffer, whose unused
entries hold -1.  Outputs are that buffer and the pair counts: whole numbers,
equal bit for bit.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

import pierce_gb300 as pg
from pierce_gb300 import batched as BT
from pierce_gb300 import capi
from pierce_gb300 import join as J
from pierce_gb300 import sizing as S

_ctx = None
_model = None


def _context() -> J.Context:
    """One context for all datasets and joins, as a program on one GPU has."""
    global _ctx
    if _ctx is None:
        _ctx = J.Context(0)
    return _ctx


def _sizing_model() -> S.SizingModel:
    global _model
    if _model is None:
        _model = S.SizingModel.load(_context(), S.TRAINED_MODEL)
    return _model


def listed():
    return [
        # the smallest call: a few dozen coarse meshes; launches and host
        # round trips are all there is
        {"name": "overlap 60 x 60", "kind": "spheres", "predicate": "overlap", "sizing": "hash", "na": 60, "nb": 60,
         "level": 2, "extent": 25.0},
        # the small benchmark configuration: 2 x 2,000 spheres, intersection
        {"name": "intersection 2000 x 2000", "kind": "spheres", "predicate": "intersection", "sizing": "hash",
         "na": 2000, "nb": 2000, "level": 3, "extent": 200.0},
        # the reference's two-pass method, odd and uneven sizes
        {"name": "two-pass 7013 x 4999", "kind": "spheres", "predicate": "overlap", "sizing": "two_pass",
         "na": 7013, "nb": 4999, "level": 3, "extent": 150.0},
        # a dense join of the sizing sweep: mixed subdivision levels, many
        # partners per mesh, table sized by the network
        {"name": "dense learned 12007 x 9001", "kind": "sweep", "predicate": "overlap", "sizing": "learned",
         "na": 12007, "nb": 9001, "partners": 20.0},
        # the float32 form in one direction over the datasets' edge lists
        {"name": "float32 one way 20000 x 15001", "kind": "float32", "predicate": "overlap", "sizing": "hash",
         "na": 20000, "nb": 15001, "level": 3},
        # the ellipsoid benchmark at full size: some meshes nested in meshes
        # of the other side, a few exact duplicates
        {"name": "intersection 50000 x 50000", "kind": "ellipsoids", "predicate": "intersection", "sizing": "hash",
         "na": 50000, "nb": 50000, "level": 3},
        {"name": "containment 50000 x 50000", "kind": "ellipsoids", "predicate": "containment", "sizing": "hash",
         "na": 50000, "nb": 50000, "level": 3},
        # long branching tubes against compact meshes (the default benchmark's
        # meshes, density and options; fewer of them)
        {"name": "tubes 128 x 6400", "kind": "tubes", "predicate": "overlap", "sizing": "learned", "na": 128,
         "nb": 6400},
        # the largest resident join, without edge lists (512 M + 128 M triangles)
        {"name": "overlap 400000 x 100000", "kind": "edgeless", "predicate": "overlap", "sizing": "hash",
         "na": 400000, "nb": 100000, "level": 3},
        # many small independent joins as one captured graph
        {"name": "batch of 64 joins", "kind": "batch", "predicate": "overlap", "sizing": "hash", "queries": 64,
         "n_lo": 10, "n_hi": 3000},
        # a query service: triangles from pinned host arrays, an intersection,
        # the pairs back, the datasets released
        {"name": "upload and join 6000 x 5003", "kind": "upload", "predicate": "intersection", "sizing": "hash",
         "na": 6000, "nb": 5003, "level": 3},
        # the command-line tools' path: whole `.pre` content with edges, own
        # hierarchies built, a fixed table
        {"name": "tool query 2000 x 1501", "kind": "tool", "predicate": "overlap", "sizing": "fixed", "na": 2000,
         "nb": 1501, "level": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spheres", "spheres", "sweep", "float32", "ellipsoids", "ellipsoids", "tubes", "edgeless",
                       "batch", "upload", "tool"])
    c = {"kind": kind, "predicate": "overlap", "sizing": "hash"}
    if kind == "spheres":
        c["predicate"] = rng.choice(["overlap", "intersection", "containment"])
        c["sizing"] = rng.choice(["hash", "two_pass"])
        c["na"], c["nb"] = _log_int(rng, 20, 20000), _log_int(rng, 20, 20000)
        c["level"] = rng.choice([2, 3])
        c["extent"] = round((c["na"] + c["nb"]) ** (1.0 / 3.0) * rng.uniform(4.0, 13.0), 3)
    elif kind == "sweep":
        c["na"], c["nb"], c["sizing"] = _log_int(rng, 1000, 20000), _log_int(rng, 1000, 20000), "learned"
        c["partners"] = round(math.exp(rng.uniform(math.log(0.5), math.log(20.0))), 3)
    elif kind in ("float32", "ellipsoids"):
        c["na"], c["nb"], c["level"] = _log_int(rng, 1000, 50000), _log_int(rng, 1000, 50000), 3
        if kind == "ellipsoids":
            c["predicate"] = rng.choice(["overlap", "intersection", "containment"])
    elif kind == "tubes":
        c["na"], c["nb"], c["sizing"] = _log_int(rng, 8, 128), _log_int(rng, 200, 6400), "learned"
    elif kind == "edgeless":
        c["na"], c["nb"] = _log_int(rng, 20000, 200000), _log_int(rng, 20000, 100000)
        c["level"] = rng.choice([2, 3])
    elif kind == "batch":
        c["queries"], c["n_lo"], c["n_hi"] = _log_int(rng, 4, 64), 10, _log_int(rng, 50, 3000)
    elif kind == "upload":
        c["predicate"] = rng.choice(["overlap", "intersection", "containment"])
        c["na"], c["nb"], c["level"] = _log_int(rng, 50, 6000), _log_int(rng, 50, 6000), rng.choice([2, 3])
    else:
        c["sizing"] = "fixed"
        c["na"], c["nb"], c["level"] = _log_int(rng, 20, 2000), _log_int(rng, 20, 2000), rng.choice([2, 3])
    return c


def _extent(n):
    """Cube side with the ellipsoid benchmark's density (50,000 in 1000^3)."""
    return 1000.0 * (n / 50000.0) ** (1.0 / 3.0)


def _ellipsoids(case, seed):
    """Instances of both sides; of B, 20 % are scaled copies inside an A mesh
    and 0.5 % exact duplicates of one."""
    hi = _extent(max(case["na"], case["nb"]))
    a = pg.instances(2 * seed + 1, case["na"], pg.ELLIPSOIDS, case["level"], p0=2.0, p1=5.0, hi=hi)
    b = pg.instances(2 * seed + 2, case["nb"], pg.ELLIPSOIDS, case["level"], p0=2.0, p1=5.0, hi=hi)
    rng = np.random.default_rng(seed)
    u, j = rng.random(len(b)), rng.integers(0, len(a), len(b))
    b[u < 0.205] = a[j[u < 0.205]]
    b["axes"][u < 0.2] *= 0.3
    return a, b


def _sweep(case, seed):
    """Mixed levels 2..4, spheres against ellipsoids, a cube side for the
    case's mean number of partners per mesh (contact shell of mean radii)."""
    ra, rb = 1.57, 3.5
    shell = 4.0 / 3.0 * math.pi * ((ra + rb) ** 3 - abs(ra - rb) ** 3)
    hi = (shell * max(case["na"], case["nb"]) / case["partners"]) ** (1.0 / 3.0)
    return (pg.instances(2 * seed + 1, case["na"], pg.SPHERES, 2, 4, hi=hi),
            pg.instances(2 * seed + 2, case["nb"], pg.ELLIPSOIDS, 2, 4, hi=hi))


def _spheres(case, seed):
    return (pg.instances(2 * seed + 1, case["na"], pg.SPHERES, case["level"], hi=case["extent"]),
            pg.instances(2 * seed + 2, case["nb"], pg.SPHERES, case["level"], hi=case["extent"]))


def _batch_opts(wave):
    return J.make_opts(predicate="overlap", expected_pairs=BT.expected_pairs(wave))


def _host_view(inst, edges):
    """A mesh view over pinned host arrays of expanded meshes; without edges
    the objects go as triangle offsets.  Returns (view, what it points to)."""
    g = pg.expand_instances(inst)
    keep, v = [], capi.MeshView()

    def pinned(a):
        t = torch.empty(max(a.nbytes, 1), dtype=torch.uint8, pin_memory=True)
        t.numpy()[:a.nbytes] = np.ascontiguousarray(a).view(np.uint8).reshape(-1)
        keep.append(t)
        return t.data_ptr()

    v.vertices, v.num_vertices = pinned(g.vertices), g.vertices.shape[0]
    v.indices, v.num_triangles = pinned(g.indices), g.num_triangles
    v.num_objects = g.num_objects
    if edges:
        v.tri_to_object = pinned(g.tri_to_object)
        v.edge_starts, v.edge_ends = pinned(g.edge_starts), pinned(g.edge_ends)
        v.edge_src, v.num_edges = pinned(g.edge_src), g.num_edges
    else:
        off = J.object_offsets(g.tri_to_object, g.num_objects)
        keep.append(off)
        v.object_offsets = off.ctypes.data
    return v, keep


def _capacity(case):
    """Pairs the caller's buffer holds: well above what these joins give."""
    if case["kind"] == "batch":
        n = 2 * case["queries"] * case["n_hi"]
    else:
        n = 4 * (case["na"] + case["nb"]) * max(1.0, case.get("partners", 1.0))
    return 1 << max(12, math.ceil(math.log2(n)))


def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    resident = J.default_tuning(defer_build=1)
    st = {"case": case, "ctx": ctx, "out": torch.full((_capacity(case), 2), -1, dtype=torch.int32, pin_memory=True)}
    if kind == "batch":
        qs = BT.workload(seed=seed, queries=case["queries"], n_lo=case["n_lo"], n_hi=case["n_hi"])
        wave = BT.make_waves(qs, budget_tris=1e12)[0]
        st["a"] = J.Dataset.from_instances(ctx, wave.a, resident)
        st["b"] = J.Dataset.from_instances(ctx, wave.b, resident)
        st["graph"] = J.JoinGraph(ctx, st["a"], st["b"], _batch_opts(wave))
        return st
    if kind in ("upload", "tool"):
        edges = kind == "tool"
        hi = _extent(max(case["na"], case["nb"]))
        a = pg.instances(2 * seed + 1, case["na"], pg.ELLIPSOIDS, case["level"], p0=2.0, p1=5.0, hi=hi)
        b = pg.instances(2 * seed + 2, case["nb"], pg.ELLIPSOIDS, case["level"], p0=2.0, p1=5.0, hi=hi)
        st["a"], st["keep_a"] = _host_view(a, edges)
        st["b"], st["keep_b"] = _host_view(b, edges)
        st["tuning"] = J.default_tuning() if edges else J.default_tuning(defer_build=1, skip_edges=1)
        st["opts"] = J.make_opts(predicate=case["predicate"], sizing=case["sizing"],
                                 hash_table_slots=1 << 20 if edges else 0)
        return st
    opts = {"predicate": case["predicate"], "sizing": case["sizing"]}
    if case["sizing"] == "learned":
        opts["sizing_model"] = _sizing_model()
    if kind == "tubes":
        hi = 1000.0 * (case["na"] / 2000.0) ** (1.0 / 3.0)
        edgeless = J.default_tuning(defer_build=1, skip_edges=1)
        g = pg.tubes(seed + 1, case["na"], 200_000, 1.0, 0.02, 0.5, 3.0, 12, 0.0, hi)
        st["a"] = J.Dataset.from_geometry(ctx, g, edgeless)
        st["b"] = J.Dataset.from_instances(
            ctx, pg.instances(seed + 2, case["nb"], pg.ELLIPSOIDS, 3, p0=2.0, p1=5.0, hi=hi), edgeless)
    else:
        if kind == "spheres":
            a, b = _spheres(case, seed)
        elif kind == "sweep":
            a, b = _sweep(case, seed)
        else:
            a, b = _ellipsoids(case, seed)
        if kind == "edgeless":
            resident = J.default_tuning(defer_build=1, skip_edges=1)
            opts["expected_pairs"] = 4 * max(case["na"], case["nb"])
        if kind == "float32":
            opts.update(precision="fp32", direction="mesh1_to_mesh2", edge_source="dataset")
        st["a"] = J.Dataset.from_instances(ctx, a, resident)
        st["b"] = J.Dataset.from_instances(ctx, b, resident)
    st["opts"] = J.make_opts(**opts)
    return st


def run(state):
    ctx, kind, out = state["ctx"], state["case"]["kind"], state["out"]
    lib = capi.lib()
    if kind == "batch":
        state["graph"].launch()
        p = state["graph"].pairs()
        out.numpy()[:len(p)] = p
        return {"pairs": out, "count": len(p)}
    if kind not in ("upload", "tool"):
        return _join_into(ctx, state["a"], state["b"], state["opts"], out)
    sets = []
    try:
        for side in ("a", "b"):
            h = C.c_void_p()
            capi.check(lib.pierce_dataset_create(ctx.handle, C.byref(state[side]), capi.HOST_MEMORY,
                                                 C.byref(state["tuning"]), C.byref(h)), "dataset_create")
            sets.append(J.Dataset(ctx, h))
        return _join_into(ctx, sets[0], sets[1], state["opts"], out)
    finally:
        for d in sets:
            d.close()


def _join_into(ctx, a, b, opts, out):
    """One join with its pairs copied into the caller's buffer."""
    lib, r, st, n, nc = capi.lib(), C.c_void_p(), capi.Stats(), C.c_uint64(), C.c_uint64()
    capi.check(lib.pierce_join(ctx.handle, a.handle, b.handle, C.byref(opts), C.byref(r), C.byref(st)), "join")
    try:
        capi.check(lib.pierce_result_count(r, C.byref(n)), "result_count")
        capi.check(lib.pierce_result_containment_count(r, C.byref(nc)), "result_containment_count")
        capi.check(lib.pierce_result_copy(ctx.handle, r, out.data_ptr(), len(out)), "result_copy")
    finally:
        lib.pierce_result_destroy(r)
    return {"pairs": out, "count": n.value, "containment": nc.value}


def _level_sizes(level):
    """(vertices, triangles) of an icosphere of this level."""
    return 10 * 4 ** level + 2, 20 * 4 ** level


def work(case):
    """Every vertex (12 bytes) and index (12 bytes per triangle) of both sides
    read once and the pairs written once (about half a pair per mesh; 20 in
    the dense sweep); one box comparison (6 operations) per triangle.  Tools
    upload edges too (28 bytes per edge)."""
    kind = case["kind"]
    if kind == "batch":
        lo, hi = math.log(case["n_lo"]), math.log(case["n_hi"])
        mean = (case["n_hi"] - case["n_lo"]) / max(hi - lo, 1e-9)
        n = 2 * case["queries"] * mean
        sizes = [_level_sizes(k) for k in range(1, 6)]
        v, t = (n * sum(s[i] for s in sizes) / len(sizes) for i in range(2))
        pairs = 0.25 * n
    elif kind == "sweep":
        n = case["na"] + case["nb"]
        sizes = [_level_sizes(k) for k in range(2, 5)]
        v, t = (n * sum(s[i] for s in sizes) / len(sizes) for i in range(2))
        pairs = case["partners"] * min(case["na"], case["nb"])
    elif kind == "tubes":
        sv, s = _level_sizes(3)
        t = 200_000 * case["na"] + s * case["nb"]
        v = 100_000 * case["na"] + sv * case["nb"]
        pairs = 0.5 * case["nb"]
    else:
        sv, s = _level_sizes(case["level"])
        n = case["na"] + case["nb"]
        v, t, pairs = sv * n, s * n, 0.25 * n
    edges = 1.5 * t if kind == "tool" else 0.0
    return {"bytes": 12.0 * v + 12.0 * t + 28.0 * edges + 8.0 * pairs, "flops": 6.0 * t}


def exact(case, seed):
    """The outputs are pairs of whole numbers: no computed values."""
    return None
