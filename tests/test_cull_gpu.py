"""Culling on both sides of the size from which chunks are walked before
their groups, and kept-group lists over more than one tile of chunks."""
import numpy as np
import pytest

import pierce_gb300 as pg
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
