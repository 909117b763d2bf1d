"""Point queries through the tree on both sides of the number of points that is
resident at once, where the kernel changes its shape: squares and containing
rects equal the oracle's, exact ties (aligned rects) and partly listed cells
included."""
import numpy as np
import pytest

import frw
import oracle as O

pytestmark = pytest.mark.gpu

WAVE = 148 * 16 * 64


@pytest.fixture(scope="module")
def aligned():
    r = np.array([[x, y, x + 12, y + 12] for x in range(20, 920, 30) for y in range(20, 920, 30)], float)
    G = O.Grid(r)
    rng = np.random.default_rng(0)
    b = G.bounds
    p = np.concatenate([rng.uniform(b[:2], b[2:], (WAVE // 2, 2)), np.round(rng.uniform(b[:2], b[2:], (WAVE, 2)))])
    return r, p, G.query_batch(p)


@pytest.mark.parametrize("cells", [(0.0, 32), (4.0, 2)])
@pytest.mark.parametrize("n", [1, 63, 64, 65, WAVE - 1, WAVE, WAVE + 1, WAVE + WAVE // 2])
def test_tree_queries_at_the_edges_of_the_shapes(aligned, cells, n):
    r, p, (sq_o, hit_o) = aligned
    with frw.Layout.from_rects(r) as L:
        L.set_cells(*cells)
        assert cells[0] == 0 or 0 < L.cells.overflow_cells < L.cells.cells
        sq, hit = L.query(p[-n:])
    assert np.array_equal(sq, sq_o[-n:]) and np.array_equal(hit, hit_o[-n:])
