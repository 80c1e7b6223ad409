"""Datasets from host arrays: object ids from ranges at the edges of a warp's
run, triangle preparation of every remainder, and hierarchies built while the
edges arrive."""
import numpy as np
import pytest
import torch

import pierce_gb300 as pg
from pierce_gb300 import capi
from pierce_gb300 import join as J
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def soup_of(counts, seed):
    """Objects of counts[o] random small triangles, three vertices each."""
    rng = np.random.default_rng(seed)
    centre = rng.uniform(0, 3, (len(counts), 1, 3)) + rng.normal(0, 0.01, (len(counts), 1, 3))
    ids = np.repeat(np.arange(len(counts)), counts).astype(np.int32)
    v = (centre[ids] + rng.uniform(-0.4, 0.4, (len(ids), 3, 3))).reshape(-1, 3).astype(np.float32)
    return v, np.arange(3 * len(ids), dtype=np.uint32).reshape(-1, 3), ids


@pytest.mark.parametrize("counts", [[1], [0, 1, 0], [127, 1], [128, 0, 0, 1], [1] * 129, [0, 0, 5, 250, 0, 1, 384, 0],
                                    [31, 33] * 40, [3] * 1000 + [0], [20000, 1, 12345]])
def test_object_ids_from_ranges(ctx, counts):
    v, idx, ids = soup_of(counts, 1)
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    none = np.zeros((0, 3), np.float32), np.zeros((0, 3), np.float32), np.zeros(0, np.int32)
    t = J.default_tuning(defer_build=1, skip_edges=1)
    ds = J.Dataset.from_arrays(ctx, v, idx, ids, *none, len(counts), tuning=t, object_offsets=off)
    assert np.array_equal(ds.download()["tri_to_object"], ids)


@pytest.mark.parametrize("counts", [[1, 2, 3], [40, 7, 90, 32, 64, 1], [5] * 70, [33] * 31, [700, 300]])
def test_prepared_triangles_join_as_the_oracle(ctx, counts):
    sides = []
    for seed in (2, 3):
        v, idx, ids = soup_of(counts, seed)
        sides.append(pg.Geometry.from_arrays(v, idx, ids).extract_edges())
    t = J.default_tuning(defer_build=1, skip_edges=1)
    got = J.overlap_join(ctx, *(J.Dataset.from_geometry(ctx, g, t) for g in sides))
    want, _ = O.overlap_keys(*sides)
    assert np.array_equal(J.pairs_to_keys(got.pairs), want)


@pytest.mark.parametrize("shuffle", [False, True])
@pytest.mark.parametrize("n", [1, 3, 60])
def test_hierarchy_built_while_the_edges_arrive(ctx, n, shuffle):
    """Pinned arrays, read in place: edges grouped by object or not."""
    sides, views, keep = [], [], []
    for seed in (4, 5):
        g = pg.icospheres(seed, n, 2, hi=1.5 * n ** (1 / 3)).extract_edges()
        p = np.random.default_rng(seed).permutation(g.num_edges) if shuffle else np.arange(g.num_edges)
        v = capi.MeshView()
        for name, a in (("vertices", g.vertices), ("indices", g.indices), ("tri_to_object", g.tri_to_object),
                        ("edge_starts", g.edge_starts[p]), ("edge_ends", g.edge_ends[p]), ("edge_src", g.edge_src[p])):
            t = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True)
            t.numpy()[:] = np.ascontiguousarray(a).view(np.uint8).reshape(-1)
            keep.append(t)
            setattr(v, name, t.data_ptr())
        v.num_vertices, v.num_triangles = g.vertices.shape[0], g.num_triangles
        v.num_edges, v.num_objects = g.num_edges, g.num_objects
        sides.append(g)
        views.append(v)
    h = [capi.C.c_void_p() for _ in views]
    t = J.default_tuning()
    for v, d in zip(views, h):
        J.check(capi.lib().pierce_dataset_create(ctx.handle, capi.C.byref(v), capi.HOST_MEMORY, capi.C.byref(t),
                                                 capi.C.byref(d)), "dataset_create")
    da, db = (J.Dataset(ctx, d) for d in h)
    want, _ = O.overlap_keys(*sides)
    for source in ("dataset", "triangles"):
        got = J.overlap_join(ctx, da, db, edge_source=source)
        assert np.array_equal(J.pairs_to_keys(got.pairs), want), source
    assert np.array_equal(J.pairs_to_keys(J.overlap_join(ctx, da, db, active_bvh=False).pairs), want)
