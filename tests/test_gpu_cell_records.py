"""Cell records at the edges of their format: cells that list up to four rects
keep them in place, longer lists go to the shared buffer (also when it has to
grow), capped cells to the tree.  Queries equal the oracle's."""
import numpy as np
import pytest

import frw
import oracle as O

pytestmark = pytest.mark.gpu


def row_of(k, side=2.0, gap=4.0):
    """k rects of one size around a centre, all about as near to it."""
    a = np.arange(k) * 2 * np.pi / k
    c = np.stack([200 + np.round(60 * np.cos(a)), 200 + np.round(60 * np.sin(a))], 1)
    return np.concatenate([c, c + side], 1)


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 6, 9, 31, 32, 33])
def test_record_of_k_rects(k):
    r = row_of(k)
    b = np.array([0.0, 0.0, 400.0, 400.0])
    rng = np.random.default_rng(k)
    p = np.concatenate([rng.uniform(0, 400, (4000, 2)), r[rng.integers(0, k, 500), :2], rng.uniform(190, 210, (500, 2))])
    ref, hit_ref = O.Grid(r, b).query_batch(p)
    with frw.Layout.from_rects(r, b) as L:
        for cells_per_rect in (16.0, 0.2, 400.0):
            L.set_cells(cells_per_rect)
            sq, hit = L.query(p)
            assert np.array_equal(sq, ref) and np.array_equal(hit, hit_ref)


def test_overlapping_rects_report_the_lowest_index():
    """Nested rects share their cells: the lowest layer index wins in a record
    and in a longer list."""
    for k in (3, 4, 5, 20):
        i = np.arange(k)[::-1, None] * 1.0  # the smallest rect has the highest index
        r = np.concatenate([100 - i, 100 - i, 110 + i, 110 + i], 1)
        b = np.array([0.0, 0.0, 220.0, 220.0])
        p = np.random.default_rng(3).uniform(70, 140, (3000, 2))
        ref, hit_ref = O.Grid(r, b).query_batch(p)
        with frw.Layout.from_rects(r, b) as L:
            sq, hit = L.query(p)
            assert np.array_equal(sq, ref) and np.array_equal(hit, hit_ref)


def test_lists_past_the_first_buffer():
    """A dense block in wide bounds: nearly every cell sees dozens of rects, more
    list entries than cells, so the lists take a second pass."""
    gx, gy = np.meshgrid(np.arange(24) * 3.0, np.arange(24) * 3.0)
    r = np.stack([gx.ravel(), gy.ravel(), gx.ravel() + 1, gy.ravel() + 1], 1) + 5000.0
    b = np.array([0.0, 0.0, 10000.0, 10000.0])
    rng = np.random.default_rng(9)
    p = np.concatenate([rng.uniform(0, 10000, (3000, 2)), rng.uniform(4990, 5090, (3000, 2))])
    ref, hit_ref = O.Grid(r, b).query_batch(p)
    with frw.Layout.from_rects(r, b) as L:
        for cells_per_rect, cap in ((0.5, 600), (16.0, 600), (200.0, 600), (200.0, 32)):
            L.set_cells(cells_per_rect, cap)
            c = L.cells
            if cap == 600:
                assert c.overflow_cells == 0 and c.entries > c.cells
            sq, hit = L.query(p)
            assert np.array_equal(sq, ref) and np.array_equal(hit, hit_ref)


@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 9])
@pytest.mark.parametrize("margin", [0.0, 2.5, 40.0, 900.0])
def test_walks_near_the_bounds(k, margin):
    """Walks of few rects in bounds from touching them to far away: cells near
    the bounds look at them, the others do not; most walks escape.  Per-walk
    records equal the oracle's for both start modes."""
    r = row_of(k)
    b = np.array([r[:, 0].min() - margin, r[:, 1].min() - margin, r[:, 2].max() + margin, r[:, 3].max() + margin])
    G = O.Grid(r, b)
    escaped = 0
    with frw.Layout.from_rects(r, b) as L:
        for o in (frw.opts(), frw.capacitance_opts(1.0)):
            for cells_per_rect in (16.0, 300.0):
                L.set_cells(cells_per_rect)
                end, hops, b1, w = L.walk_trace(k - 1, 0, 3000, 11, o)
                cfg = G.walk_cfg(target=k - 1, gauss_mode=o.gauss_mode, gauss_param=o.gauss_param,
                                 start_mode=o.start_mode, hop_cap=o.hop_cap, seed=11)
                ref = G.walks(cfg, 0, 3000)
                for x, y in zip((end, hops, b1, w), ref):
                    assert np.array_equal(x, y)
                escaped += int((end == -1).sum())
    assert escaped > 0


@pytest.mark.parametrize("cells_per_rect", [0.2, 1.0, 16.0, 400.0, 20000.0])
@pytest.mark.parametrize("kind", ["alone", "pair", "ring", "nested", "columns", "layer"])
def test_nearest_other_conductor(kind, cells_per_rect):
    """The nearest conductor other than the target, in the control variate's
    features: in the lists of the cells around the point, near or at the
    bounds' cells, several rings away, beyond them (the tree) or nowhere."""
    b = np.array([0.0, 0.0, 400.0, 400.0])
    r = {"alone": np.array([[200.0, 200, 210, 210]]),
         "pair": np.array([[3.0, 3, 8, 8], [380.0, 390, 390, 397]]),
         "ring": row_of(33),
         "nested": np.array([[100.0, 100, 200, 200], [120.0, 120, 140, 140], [90.0, 90, 210, 210]]),
         "columns": np.array([[x, y, x + 10, y + 10] for x in range(20, 380, 30) for y in range(20, 380, 30)], float),
         "layer": frw.generate_layout(5, 16, 400.0).astype(np.float64)}[kind]
    rng = np.random.default_rng(len(r))
    t = r[0]
    p = np.concatenate([rng.uniform(0, 400, (600, 2)), rng.uniform(t[:2] - 3, t[2:] + 3, (600, 2)),
                        np.round(rng.uniform(0, 400, (300, 2)))]).clip(0, 400)
    rec = np.zeros((len(p), 4))
    rec[:, :2] = p
    rec[:, 2] = rng.choice([1.0, 2.5, 7.0], len(p))
    with frw.Layout.from_rects(r, b) as L:
        L.set_cells(cells_per_rect)
        got = L.cv_features(0, rec)
    assert np.array_equal(got, O.cv_features(r, 0, rec))


@pytest.mark.parametrize("width", [60, 200, 900, 4000])
def test_coarse_lists_longer_than_their_room(width):
    """Long thin rects on a grid built through coarse cells: few rects per
    coarse cell, more than there is room for at first (the pass runs again),
    and more than a coarse cell keeps (its cells take them from the tree)."""
    n = 4200
    y = np.arange(n) * 4.0
    r = np.stack([np.zeros(n), y, np.full(n, float(width)), y + 2], 1)
    b = np.array([-50.0, -50.0, width + 50.0, 4.0 * n + 50.0])
    rng = np.random.default_rng(width)
    p = np.concatenate([rng.uniform(b[:2], b[2:], (4000, 2)), np.round(rng.uniform(b[:2], b[2:], (1000, 2)))])
    ref, hit_ref = O.Grid(r, b).query_batch(p)
    with frw.Layout.from_rects(r, b) as L:
        sq, hit = L.query(p)
    assert np.array_equal(sq, ref) and np.array_equal(hit, hit_ref)
