"""The GPU tree build against the oracle's restatement of it, bit for bit, at
the sizes where its kernels change what they do: a root that is a leaf, leaves
cut off by the depth, equal positions, one particle past a leaf's capacity, and
particle counts around the 1024-particle blocks."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _positions(pkg, kind, n):
    rng = np.random.default_rng(n)
    if kind == "plummer":
        return pkg.ic.make_plummer(n, seed=n)
    if kind == "impact":
        return pkg.ic.make_impact(n - n // 5, n // 5, seed=n)
    ic = pkg.ic.make_cube(n, seed=n)
    if kind == "doubled":  # every position many times: deeper than the keys can tell
        ic["pos"] = np.ascontiguousarray(ic["pos"][rng.integers(0, max(n // 50, 1), n)])
    return ic


@pytest.mark.parametrize("kind,n,leaf,depth", [
    ("cube", 1, 4, 7), ("cube", 4, 4, 7), ("cube", 5, 4, 7), ("cube", 33, 32, 7), ("cube", 1023, 1, 7),
    ("cube", 1024, 4, 10), ("cube", 1025, 32, 1), ("doubled", 3000, 1, 7), ("doubled", 2049, 16, 3),
    ("plummer", 20000, 4, 10), ("plummer", 70001, 32, 10), ("impact", 30000, 1, 7), ("impact", 30001, 100000, 7),
    ("impact", 250001, 32, 7),
])
def test_tree_matches_the_oracle(cuda, pkg, O, kind, n, leaf, depth):
    ic = _positions(pkg, kind, n)
    want = O.tree_morton(ic["pos"], leaf, depth)
    with pkg.Compute(ic, max_children_in_leaf=leaf, max_tree_depth=depth) as c:
        for _ in range(2):  # the second build finds the first one's scratch
            got = c.get_tree()
            assert got["n_nodes"] == want["n_nodes"] and got["n_levels"] == want["n_levels"]
            for k in ("tree", "level_offsets", "level_nodes"):
                assert np.array_equal(got[k], want[k]), k
            c.updateOctreeBuffer()
        c.synchronize()
        assert c.health() == 0
