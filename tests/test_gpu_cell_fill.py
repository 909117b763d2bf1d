"""Cell lists longer than the buffer the records pass has room for: they are
written by the pass that follows.  Queries over them equal the oracle's and the
tree's, on grids built from the tree and through coarse cells, with lists that
straddle the room's end, lists cut off by max_per_cell and cells near the bounds."""
import numpy as np
import pytest

import frw
import oracle as O

pytestmark = pytest.mark.gpu


def overlapping(n, size, seed=2):
    rng = np.random.default_rng(seed)
    a = rng.uniform(0, 100.0 * n**0.5, (n, 2))
    e = rng.uniform(size / 2, size, (n, 2))
    return np.concatenate([a, a + e], 1).astype(np.float32)


# rects, their size, cells per rect, max_per_cell: one-level grids below 65,536 cells, coarse cells above
@pytest.mark.parametrize("n,size,per,cap", [(3000, 600.0, 1.0, 200), (300, 700.0, 16.0, 200), (2000, 300.0, 8.0, 64),
                                            (6000, 300.0, 16.0, 32), (6000, 400.0, 16.0, 14), (6000, 270.0, 12.0, 32)])
def test_lists_past_the_room(n, size, per, cap):
    r = overlapping(n, size)
    rng = np.random.default_rng(n)
    with frw.Layout.from_rects(r) as L:
        b = L.bounds
        p = np.concatenate([rng.uniform(b[:2], b[2:], (30_000, 2)), np.round(rng.uniform(b[:2], b[2:], (10_000, 2))),
                            r[rng.integers(0, n, 5000), :2].astype(float)]).clip(b[:2], b[2:])
        L.set_cells(0)
        sq_t, hit_t = L.query(p)
        L.set_cells(per, cap)
        c = L.cells
        # the lists end past the room: cells without one have four rects at most
        assert c.entries > 4 * c.cells + max(c.cells // 2, 4096)
        assert (cap == 14) == (c.overflow_cells > 0)
        sq, hit = L.query(p)
        assert np.array_equal(sq, sq_t) and np.array_equal(hit, hit_t)
        end, hops, b1, w = L.walk_trace(1, 0, 2000, 5, frw.capacitance_opts(1.0))
    G = O.Grid(r.astype(np.float64), b)
    sq_o, hit_o = G.query_batch(p[::9])
    assert np.array_equal(sq[::9], sq_o) and np.array_equal(hit[::9], hit_o)
    cfg = G.walk_cfg(target=1, gauss_mode=frw.GAUSS_OFFSET, gauss_param=1.0, start_mode=frw.START_UNIFORM, seed=5)
    for x, y in zip((end, hops, b1, w), G.walks(cfg, 0, 2000)):
        assert np.array_equal(x, y)
