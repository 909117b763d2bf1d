"""Trees of layouts past the one-block build: sizes around its limit, deep trees
(clusters, equal keys split by index) and their queries without cell lists."""
import numpy as np
import pytest

import frw
import oracle as O

pytestmark = pytest.mark.gpu


def check(r, bounds=None, n=4000):
    r = r.astype(np.float64)
    G = O.Grid(r, bounds)
    b = G.bounds
    rng = np.random.default_rng(len(r))
    i = rng.integers(0, len(r), n // 2)
    p = np.concatenate([np.stack([rng.uniform(b[0], b[2], n), rng.uniform(b[1], b[3], n)], 1),
                        r[i, :2] + rng.uniform(-3, 3, (n // 2, 2))])
    ref, hit_ref = G.query_batch(p)
    with frw.Layout.from_rects(r.astype(np.float32), bounds) as L:
        info = L.info
        sq, hit = L.query(p)
        L.set_cells(0)  # the tree alone
        sq_t, hit_t = L.query(p)
    assert np.array_equal(sq, ref) and np.array_equal(hit, hit_ref)
    assert np.array_equal(sq_t, ref) and np.array_equal(hit_t, hit_ref)
    return info


@pytest.mark.parametrize("n", [65_535, 65_536, 65_537, 131_071, 300_001])
def test_sizes_around_the_one_block_build(n):
    info = check(frw.generate_layout(n, n, 100 * n**0.5))
    assert 7 <= info.depth <= 12 and info.n_nodes >= n // 32


def test_deep_trees():
    """70,000 small rects in one corner of wide bounds: many levels re-split in
    one quadrant before the first node that branches."""
    k = np.arange(70_000)
    x, y = (k % 265) * 2.0, (k // 265) * 2.0
    info = check(np.stack([x, y, x + 1, y + 1], 1), np.array([0.0, 0.0, 1e6, 1e6]))
    assert info.depth >= 6


def test_equal_keys_are_split_by_index():
    """Rects of one centre cell (equal Morton keys) by the thousand."""
    k = np.arange(66_000)
    x, y = (k % 300) * 0.015625, (k // 300) * 0.015625
    r = np.stack([x, y, x + 0.0078125, y + 0.0078125], 1)
    check(r, np.array([0.0, 0.0, 500_000.0, 500_000.0]), n=600)
