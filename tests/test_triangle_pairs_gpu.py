"""Joins by triangle pairs (exact two-way joins whose sides take their rays
from the kept triangles) against the CPU oracle and against the per-ray walk
over the binary nodes, which traces segments."""
import numpy as np
import pytest

import pierce_gb300 as pg
from pierce_gb300 import join as J
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def duplicates(seed=3):
    """Half of B's meshes are A's: shared vertices and coplanar faces."""
    a = pg.instances(seed, 60, pg.ELLIPSOIDS, 2, p0=1.0, p1=2.0, hi=14.0)
    b = pg.instances(seed + 1, 50, pg.ELLIPSOIDS, 2, p0=1.0, p1=2.0, hi=14.0)
    b[:25] = a[:25]
    return pg.expand_instances(a), pg.expand_instances(b)


def coarse_and_fine():
    """Two coarse meshes whose groups meet thousands of the leaves of fine
    ones: walks longer than one round's budget."""
    a = pg.instances(7, 6, pg.SPHERES, 6, p0=float(np.log(3.0)), p1=0.05, hi=4.0)
    b = pg.instances(8, 2, pg.SPHERES, 0, p0=float(np.log(3.0)), p1=0.05, hi=4.0)
    return pg.expand_instances(a), pg.expand_instances(b)


def degenerate():
    """Zero-area triangles (a repeated vertex, collinear vertices) among
    whole ones, and groups that mix objects of one to five triangles."""
    rng = np.random.default_rng(5)

    def side():
        v, idx, obj = [], [], []
        for o in range(120):
            c = rng.uniform(0, 6, 3)
            for _ in range(rng.integers(1, 6)):
                p = c + rng.uniform(-1, 1, (3, 3))
                kind = rng.integers(0, 8)
                if kind == 0:
                    p[2] = p[1]
                elif kind == 1:
                    p = np.round(p * 4) / 4
                    p[2] = 2 * p[1] - p[0]
                idx.append([len(v), len(v) + 1, len(v) + 2])
                v.extend(p)
                obj.append(o)
        g = pg.Geometry.from_arrays(np.array(v, np.float32), np.array(idx, np.uint32), np.array(obj, np.int32))
        return g
    return side(), side()


CASES = {"one group": lambda: (pg.icospheres(1, 1, 1, hi=0.0), pg.icospheres(2, 1, 1, hi=0.0)),
         "odd sizes": lambda: (pg.icospheres(101, 67, 2, hi=20.0), pg.icospheres(202, 31, 3, hi=20.0)),
         "duplicates": duplicates, "coarse and fine": coarse_and_fine, "degenerate": degenerate}


@pytest.mark.parametrize("leaf", [1, 2, 4, 8, 16])
@pytest.mark.parametrize("name", sorted(CASES))
def test_triangle_pairs_match_oracle_and_rays(ctx, name, leaf):
    A, B = CASES[name]()
    for g in (A, B):
        if not g.has_edges:
            g.extract_edges()
    t = J.default_tuning(defer_build=1, skip_edges=1)
    da, db = J.Dataset.from_geometry(ctx, A, t), J.Dataset.from_geometry(ctx, B, t)
    want, _ = O.overlap_keys(A, B)
    # exact inline: a full queue of deferred tests would trace (and count) every ray again
    rays = J.overlap_join(ctx, da, db, leaf_size=leaf, traversal="per_ray_binary", defer_exact=False)
    for defer in (True, False):
        got = J.overlap_join(ctx, da, db, leaf_size=leaf, defer_exact=defer)
        assert np.array_equal(J.pairs_to_keys(got.pairs), want), (name, leaf, defer)
        assert np.array_equal(got.pairs, rays.pairs)
        assert defer or got.stats["rays"] == rays.stats["rays"]
        assert got.stats["active_triangles"] == rays.stats["active_triangles"]
    inter = J.intersection_join(ctx, da, db, leaf_size=leaf)
    assert np.array_equal(J.pairs_to_keys(inter.pairs), O.intersection_keys(A, B))


def test_triangle_pairs_of_interleaved_objects(ctx):
    """Triangles in random order: every group mixes objects."""
    A, B = pg.icospheres(5, 40, 2, hi=14.0), pg.icospheres(6, 45, 2, hi=14.0)
    rng = np.random.default_rng(1)
    sides = []
    for G in (A, B):
        p = rng.permutation(G.num_triangles)
        sides.append(pg.Geometry.from_arrays(G.vertices, G.indices[p], G.tri_to_object[p]).extract_edges())
    t = J.default_tuning(defer_build=1, skip_edges=1)
    got = J.overlap_join(ctx, *(J.Dataset.from_geometry(ctx, g, t) for g in sides))
    want, _ = O.overlap_keys(A, B)
    assert np.array_equal(J.pairs_to_keys(got.pairs), want) and len(want) > 10


def test_triangle_pairs_into_small_tables(ctx):
    """A table that fills up is enlarged and the pairs found again."""
    A, B = duplicates(11)
    t = J.default_tuning(defer_build=1, skip_edges=1)
    da, db = J.Dataset.from_geometry(ctx, A, t), J.Dataset.from_geometry(ctx, B, t)
    want, _ = O.overlap_keys(A, B)
    got = J.overlap_join(ctx, da, db, sizing="fixed", hash_table_slots=16, max_retries=8)
    assert np.array_equal(J.pairs_to_keys(got.pairs), want) and got.stats["retries"] > 0
