"""Culling on both sides of the size from which chunks are walked before
their groups, and kept-group lists over more than one tile of chunks."""
import numpy as np
import pytest

import pierce_gb300 as pg
from pierce_gb300 import capi
from pierce_gb300 import join as J
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("meshes", [(3, 60), (700, 900), (900, 40)])
def test_culled_joins_match_the_oracle(ctx, meshes):
    """0.004 to 1.15 M triangles a side, nearly all of active objects."""
    sides = [pg.icospheres(21 + k, n, 3, hi=2.2 * max(meshes) ** (1 / 3)).extract_edges() for k, n in enumerate(meshes)]
    t = J.default_tuning(defer_build=1, skip_edges=1)
    da, db = (J.Dataset.from_geometry(ctx, g, t) for g in sides)
    want, _ = O.overlap_keys(*sides)
    for leaf in (1, 4, 16):
        got = J.overlap_join(ctx, da, db, leaf_size=leaf)
        assert np.array_equal(J.pairs_to_keys(got.pairs), want), leaf
    rays = J.overlap_join(ctx, da, db, sizing="two_pass")
    assert np.array_equal(J.pairs_to_keys(rays.pairs), want) and len(want) > 10


@pytest.mark.parametrize("predicate", ["overlap", "intersection"])
@pytest.mark.parametrize("n,level", [(40, 1), (40, 5), (90, 5)])
def test_two_pass_keys_by_set_and_by_sort(ctx, n, level, predicate):
    """A few thousand and a million raw keys (kept in the pair set) and over
    four million (sorted), nearly all of them repeats."""
    A, B = (pg.icospheres(31 + k, n, level, hi=1.2, ln_mu=0.0, sigma=0.05).extract_edges() for k in range(2))
    da, db = J.Dataset.from_geometry(ctx, A), J.Dataset.from_geometry(ctx, B)
    if predicate == "intersection":
        # more odd parity pairs than a two-pass join keeps (8 per object)
        with pytest.raises(capi.PierceError, match="parity output overflow"):
            J.join(ctx, da, db, predicate=predicate, sizing="two_pass")
        return
    got = J.join(ctx, da, db, predicate=predicate, sizing="two_pass")
    assert (sum(got.stats["raw_pairs"]) > 1 << 22) == (n == 90)
    assert np.array_equal(J.pairs_to_keys(got.pairs), O.overlap_keys(A, B)[0])


@pytest.mark.parametrize("n", [2, 300, 2000])
def test_two_pass_intersections_within_their_room(ctx, n):
    A, B = (pg.icospheres(51 + k, n, 2, hi=3.5 * n ** (1 / 3), ln_mu=0.2, sigma=0.5).extract_edges() for k in range(2))
    for x, y in ((A, B), (B, A)):
        got = J.intersection_join(ctx, J.Dataset.from_geometry(ctx, x), J.Dataset.from_geometry(ctx, y), sizing="two_pass")
        assert np.array_equal(J.pairs_to_keys(got.pairs), O.intersection_keys(x, y))


@pytest.mark.parametrize("direction", ["mesh1_to_mesh2", "mesh2_to_mesh1"])
@pytest.mark.parametrize("source", ["dataset", "triangles"])
def test_one_way_joins_list_their_side_only(ctx, direction, source):
    A, B = (pg.icospheres(41 + k, 200, 2, hi=9.0).extract_edges() for k in range(2))
    da, db = J.Dataset.from_geometry(ctx, A), J.Dataset.from_geometry(ctx, B)
    for sizing in ("hash", "two_pass"):
        got = J.overlap_join(ctx, da, db, direction=direction, sizing=sizing, edge_source=source)
        plain = J.overlap_join(ctx, da, db, direction=direction, sizing=sizing, cull_objects=False, active_bvh=False)
        assert np.array_equal(got.pairs, plain.pairs) and len(got.pairs) > 20
