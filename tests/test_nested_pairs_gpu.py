"""Nested and crossing spheres of every pairing of 20 to 5,120 triangles:
patches on both sides of what a warp keeps, pairs decided by a warp, by a
block, and after an empty, a small and a whole patch, in both directions."""
import numpy as np
import pytest

import pierce_gb300 as pg
from pierce_gb300 import join as J
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


def nested(levels, others, seed=9):
    """One A and one B per pairing of levels and placement, 4 apart."""
    rng = np.random.default_rng(seed)
    # radius of B and distance of its centre: concentric, inside, crossing, just inside, around
    places = [(0.3, 0.0), (0.3, 0.6), (0.3, 0.75), (0.02, 0.9), (0.9, 0.01), (1.0, 0.0), (1.2, 0.02)]
    rows = [(la, lb, r, d) for la in levels for lb in others for r, d in places]
    a = pg.instances(1, len(rows), pg.SPHERES, 2, p0=0.0, p1=0.0, hi=0.0)
    b = a.copy()
    for i, (la, lb, r, d) in enumerate(rows):
        u = rng.normal(size=3)
        at = 4.0 * np.array([i % 6, i // 6 % 6, i // 36], float)
        a["center"][i], a["level"][i] = at, la
        b["center"][i], b["level"][i], b["axes"][i] = at + d * u / np.linalg.norm(u), lb, r
    return pg.expand_instances(a), pg.expand_instances(b)


@pytest.mark.parametrize("levels,others", [([0, 1, 2], [0, 1, 2, 3]), ([3, 4], [0, 2]), ([0, 2], [3, 4]), ([4], [4])])
def test_nested_pairs_match_oracle(ctx, levels, others):
    A, B = nested(levels, others)
    want, inter = O.containment_keys(A, B), O.intersection_keys(A, B)
    assert 0 < len(want) < len(inter)
    da, db = J.Dataset.from_geometry(ctx, A), J.Dataset.from_geometry(ctx, B)
    for sizing in ("hash", "two_pass"):
        got = J.containment_join(ctx, da, db, sizing=sizing)
        assert np.array_equal(J.pairs_to_keys(got.pairs), want), sizing
    assert np.array_equal(J.pairs_to_keys(J.containment_join(ctx, db, da).pairs), O.containment_keys(B, A))
    assert np.array_equal(J.pairs_to_keys(J.intersection_join(ctx, da, db).pairs), inter)


@pytest.mark.parametrize("n", [1, 31, 33, 130])
def test_parity_of_few_and_many_objects(ctx, n):
    """Sources that are a part of a warp, more than one, more than a block."""
    A, B = pg.icospheres(n, 1, 3, hi=0.0, ln_mu=2.0, sigma=0.0), pg.icospheres(n + 1, n, 1, ln_mu=-1.0, sigma=0.1,
                                                                               lo=-5.0, hi=5.0)
    for x, y in ((A, B), (B, A)):
        dx, dy = J.Dataset.from_geometry(ctx, x), J.Dataset.from_geometry(ctx, y)
        assert np.array_equal(J.pairs_to_keys(J.containment_join(ctx, dx, dy).pairs), O.containment_keys(x, y))
        assert np.array_equal(J.pairs_to_keys(J.intersection_join(ctx, dx, dy).pairs), O.intersection_keys(x, y))
