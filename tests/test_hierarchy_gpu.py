"""Hierarchies at the edges of a build tile (512 positions), over more tiles
than are looked through one by one, with collapsed leaves across tiles and
with positions that share a code."""
import numpy as np
import pytest

import pierce_gb300 as pg
from pierce_gb300 import join as J
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def triangles(n, kind, seed, per_object=4, size=0.2):
    """n triangles over a cube: spread, in one place, or along a sheet."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, 10, (n, 1, 3))
    if kind == "one place":
        c = np.repeat(rng.uniform(0, 10, (1, 1, 3)), n, axis=0)
    elif kind == "sheet":
        c[:, 0, 1:] = np.round(c[:, 0, 1:2] / 10) * 7
    v = (c + rng.uniform(-size, size, (n, 3, 3))).reshape(-1, 3).astype(np.float32)
    return pg.Geometry.from_arrays(v, np.arange(3 * n, dtype=np.uint32).reshape(-1, 3),
                                   (np.arange(n) // per_object).astype(np.int32)).extract_edges()


@pytest.mark.parametrize("kind", ["spread", "one place", "sheet"])
@pytest.mark.parametrize("n,leaf", [(2, 1), (511, 1), (512, 4), (513, 1), (514, 8), (1024, 1), (1025, 3), (5000, 16),
                                    (65536, 1), (65537, 1)])
def test_own_hierarchies_find_the_oracles_pairs(ctx, n, leaf, kind):
    A, B = triangles(n, kind, 1, size=0.3), triangles(60, "spread", 2, size=6.0)
    t = J.default_tuning(leaf_size=leaf)
    da, db = J.Dataset.from_geometry(ctx, A, t), J.Dataset.from_geometry(ctx, B, t)
    info = da.info()
    used = A.vertices[A.indices.reshape(-1)]
    assert np.array_equal(np.array(info.bounds_lo[:], np.float32), used.min(0))
    assert np.array_equal(np.array(info.bounds_hi[:], np.float32), used.max(0))
    want, _ = O.overlap_keys(A, B)
    for traversal in ("per_ray", "per_ray_binary"):
        got = J.overlap_join(ctx, da, db, active_bvh=False, cull_objects=False, leaf_size=leaf, traversal=traversal)
        assert np.array_equal(J.pairs_to_keys(got.pairs), want), traversal
    assert np.array_equal(J.pairs_to_keys(J.overlap_join(ctx, da, db, leaf_size=leaf).pairs), want)


def test_a_hierarchy_of_many_tiles(ctx):
    """More than 256 tiles: nodes find their boxes by super tiles."""
    A, B = triangles(300000, "spread", 3, per_object=20), triangles(40, "spread", 4)
    t = J.default_tuning(leaf_size=1)
    da, db = J.Dataset.from_geometry(ctx, A, t), J.Dataset.from_geometry(ctx, B, t)
    want, _ = O.overlap_keys(A, B)
    got = J.overlap_join(ctx, da, db, active_bvh=False, cull_objects=False)
    assert np.array_equal(J.pairs_to_keys(got.pairs), want) and len(want) > 10
