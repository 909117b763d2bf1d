"""Layouts whose cell lists need the builds' second passes, with the list lengths
worked out on the host to show that they do: coarse lists longer in all than
their first room, coarse cells past their cap, and 3-D lists past ten entries a
cell.  Queries equal the oracle's."""
import numpy as np
import pytest

import frw
import oracle as O

pytestmark = pytest.mark.gpu

COARSE, ROOM, CAP, TWO_LEVELS = 4, 12, 64, 1 << 16  # cells per side, entries per coarse cell, rects, cells


def coarse_lists(r, b, c):
    """Rects per coarse cell: those touching it grown by its centre's clearance and half a side."""
    side = COARSE * c.cell_side
    ix, iy = np.meshgrid(np.arange(-(-c.nx // COARSE)), np.arange(-(-c.ny // COARSE)))
    x0, y0 = b[0] + ix.ravel() * side, b[1] + iy.ravel() * side
    x, y = x0 + side / 2, y0 + side / 2
    d = np.minimum(np.minimum(x - b[0], b[2] - x), np.minimum(y - b[1], b[3] - y))
    n = np.empty(len(x), np.int64)
    for k in range(0, len(x), 500):
        s = slice(k, k + 500)
        gap = np.maximum(np.maximum(r[None, :, 0] - x[s, None], x[s, None] - r[None, :, 2]),
                         np.maximum(r[None, :, 1] - y[s, None], y[s, None] - r[None, :, 3])).min(1)
        g = np.maximum(np.minimum(gap, d[s]), 0) + side / 2
        n[s] = ((r[None, :, 2] >= (x0[s] - g)[:, None]) & (r[None, :, 0] <= (x0[s] + side + g)[:, None]) &
                (r[None, :, 3] >= (y0[s] - g)[:, None]) & (r[None, :, 1] <= (y0[s] + side + g)[:, None])).sum(1)
    return n


@pytest.mark.parametrize("width,past_room,past_cap", [(200, True, False), (900, True, False), (6000, False, True)])
def test_coarse_lists(width, past_room, past_cap):
    n = 4200
    y = np.arange(n) * 4.0
    r = np.stack([np.zeros(n), y, np.full(n, float(width)), y + 2], 1)
    b = np.array([-50.0, -50.0, width + 50.0, 4.0 * n + 50.0])
    rng = np.random.default_rng(width)
    p = np.concatenate([rng.uniform(b[:2], b[2:], (4000, 2)), np.round(rng.uniform(b[:2], b[2:], (1000, 2)))])
    with frw.Layout.from_rects(r, b) as L:
        c = L.cells
        sq, hit = L.query(p)
    assert c.cells >= TWO_LEVELS
    m = coarse_lists(r, b, c)
    assert (m[m <= CAP].sum() > 1.05 * ROOM * len(m)) == past_room
    assert ((m > CAP + 2).sum() > len(m) // 10) == past_cap
    ref, hit_ref = O.Grid(r, b).query_batch(p)
    assert np.array_equal(sq, ref) and np.array_equal(hit, hit_ref)


@pytest.mark.parametrize("cells_per_box", [0.05, 0.4, 1.0])
def test_lists3_past_ten_entries_a_cell(cells_per_box):
    g = np.stack(np.meshgrid(*[np.arange(14)] * 3, indexing="ij"), -1).reshape(-1, 3) * 2.5
    b = np.concatenate([g, g + 2.0], 1).astype(np.float32)
    B = O.Boxes3(b, grid=True)
    rng = np.random.default_rng(0)
    p = B.bounds[:3] + rng.random((8000, 3)) * (B.bounds[3:] - B.bounds[:3])
    p[:2000] = np.round(p[:2000] * 4) / 4
    p = p.clip(B.bounds[:3], B.bounds[3:])
    with frw.Layout3.from_boxes(b, None, cells_per_box) as L:
        i = L.info
        d, k = L.query(p)
    assert i.levels == 1 and i.list_entries > 10 * np.prod(i.grid[:]) + 4096
    d_o, k_o = B.nearest(p)
    assert np.array_equal(d, d_o) and np.array_equal(k, k_o)
