"""Joins with an exact number of pairs: the order of the result at the sizes
where its sort changes form, and the pair table used again after it."""
import numpy as np
import pytest

import pierce_gb300 as pg
from pierce_gb300 import join as J

pytestmark = pytest.mark.gpu


def crossing(n, seed=1):
    """n triangles and n others that each cross one of them, in any order."""
    side = int(np.ceil(n ** (1 / 3)))
    i = np.arange(n)
    at = 3.0 * np.stack([i % side, i // side % side, i // side ** 2], 1)[:, None, :]
    a = at + np.array([[0, 0, 0], [1, 0, 0], [0, 1, 0]], float)
    b = at + np.array([[0.2, 0.2, -0.5], [0.2, 0.2, 0.5], [0.3, 0.2, 0.5]], float)
    p = np.random.default_rng(seed).permutation(n)  # B's object k crosses A's p[k]
    idx = np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    A = pg.Geometry.from_arrays(a.reshape(-1, 3).astype(np.float32), idx, i.astype(np.int32)).extract_edges()
    B = pg.Geometry.from_arrays(b[p].reshape(-1, 3).astype(np.float32), idx, i.astype(np.int32)).extract_edges()
    want = np.empty(n, np.int64)
    want[p] = i
    return A, B, want


@pytest.mark.parametrize("n", [1, 31, 32, 33, 2047, 2048, 2049, 16384, 16385])
def test_pairs_come_in_order(ctx, n):
    A, B, want = crossing(n)
    da, db = J.Dataset.from_geometry(ctx, A), J.Dataset.from_geometry(ctx, B)
    keys = (np.arange(n, dtype=np.uint64) << np.uint64(32)) | want.astype(np.uint64)
    for kw in (dict(), dict(sizing="two_pass"), dict(), dict(sizing="fixed", hash_table_slots=1 << 16)):
        got = J.overlap_join(ctx, da, db, **kw)
        assert np.array_equal(J.pairs_to_keys(got.pairs), keys), kw
