"""3-D clearance queries where the FP32 screen of a cell's list can go wrong:
exact and near ties between boxes, touching boxes, coordinates up to 2^23, odd
list lengths, points on boxes.  Points lie inside the bounds: a cell's list
holds the nearest box of its own points, and points outside take the clamped
cell's."""
import numpy as np
import pytest

import frw
import oracle as O

pytestmark = pytest.mark.gpu


def boxes_at(scale, shift, k):
    """k^3 equal boxes on a grid (every plane between two of them ties) moved to
    `shift`, one of them a hair smaller."""
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3) * 3.0 * scale + shift
    b = np.concatenate([g, g + 2.0 * scale], 1).astype(np.float32)
    b[0, 3] = np.nextafter(b[0, 3], np.float32(-np.inf))
    return b


@pytest.mark.parametrize("scale,shift,k", [(1.0, 0.0, 1), (1.0, 0.0, 2), (0.37, 0.0, 5), (8.0, 8388000.0, 4), (1000.0, -8388000.0, 6),
                                           (1e-3, 1.0, 3)])
@pytest.mark.parametrize("cells_per_box", [0.3, 8.0, 64.0])
def test_near_ties(scale, shift, k, cells_per_box):
    b = boxes_at(scale, shift, k)
    rng = np.random.default_rng(k)
    lo, hi = b[:, :3].min(0).astype(float) - scale, b[:, 3:].max(0).astype(float) + scale
    p = lo + rng.random((6000, 3)) * (hi - lo)
    mid = b[rng.integers(0, len(b), 2000), 3:].astype(float) + 0.5 * scale  # half way to the next box
    p[:2000] = mid * (1 + rng.choice([0, 1e-16, 1e-12, -1e-9, 1e-7, 1e-6], (2000, 1)))
    p[2000:2500] = b[rng.integers(0, len(b), 500), :3]  # corners
    bounds = np.concatenate([np.minimum(lo, p.min(0)) - scale, np.maximum(hi, p.max(0)) + scale])
    d_o, k_o = O.Boxes3(b).nearest(p)
    with frw.Layout3.from_boxes(b, bounds, cells_per_box) as L:
        d, near = L.query(p)
    assert np.array_equal(d, d_o) and np.array_equal(near, k_o)


def test_touching_boxes_and_points_not_finite():
    x = np.arange(9) * 4.0
    b = np.stack([x, 0 * x, 0 * x, x + 4, 0 * x + 5, 0 * x + 5], 1).astype(np.float32)  # a bar of nine boxes
    rng = np.random.default_rng(1)
    p = np.concatenate([np.stack([rng.uniform(-5, 41, 3000), rng.uniform(-9, 14, 3000), rng.uniform(-9, 14, 3000)], 1),
                        np.stack([x, 0 * x + 7, 0 * x + 2], 1)])  # above the seams
    d_o, k_o = O.Boxes3(b).nearest(p)
    with frw.Layout3.from_boxes(b, [-6, -10, -10, 42, 15, 15]) as L:
        d, near = L.query(p)
        inf, _ = L.query(np.array([[np.inf, 0, 0], [1e300, 2, 2], [0, -np.inf, 0]]))
    assert np.array_equal(d, d_o) and np.array_equal(near, k_o)
    assert np.array_equal(inf, [np.inf, 1e300 - 36.0, np.inf])


@pytest.mark.parametrize("walks", [1, 31, 33, 255, 257, 4097, 200_001, 400_003])
def test_walk_counts_and_launch_shapes(walks):
    """Every launch shape (one block or many, claims of 32 or 128, thresholds in
    shared memory or not) runs the same walks."""
    b = frw.generate_layout3(21, 300, 350.0, 400.0, 5, 50, 5, 20, 2)
    with frw.Layout3.from_boxes(b) as L:
        r = L.walk(3, walks, 5)
        s = L.walk(3, walks, 5, frw.opts3(blocks_per_sm=1, refill_min=1))
        end, hops, _, w = L.walk_trace(3, 0, walks, 5)
    assert r.hops_total == s.hops_total == int(hops.sum()) and r.escaped == s.escaped == int((end == -1).sum())
    assert np.array_equal(r.conductor, s.conductor) and np.array_equal(r.hits, s.hits)
    k, n = np.unique(end[end >= 0], return_counts=True)
    assert np.array_equal(r.conductor, k) and np.array_equal(r.hits, n)
    assert np.allclose(r.sum_w, [w[end == c].sum() for c in k], rtol=1e-11, atol=1e-11 * np.abs(w).sum())


@pytest.mark.parametrize("k,step", [(3, 0), (4, 0), (7, 0), (9, 0), (9, 1e-7), (9, 1e-3)])
def test_long_lists_of_ties(k, step):
    """A block of aligned boxes in wide bounds: the lists of distant cells hold
    all of it (from 27 entries, scanned again on ties, to 729, compared on the
    spot), and whole faces of it tie, exactly or nearly.  Queries and walks."""
    b = boxes_at(1.0, 0.0, k)
    b[1:, :3] += np.float32(step) * np.arange(len(b) - 1, dtype=np.float32)[:, None] / len(b)
    bounds = np.array([-300.0, -250, -200, 300, 320, 280])
    rng = np.random.default_rng(k)
    p = bounds[:3] + rng.random((5000, 3)) * (bounds[3:] - bounds[:3])
    p[:2000] = np.round(p[:2000])
    p[2000:2500] = 1.5 * k + rng.choice([-150.0, 150.0], (500, 3))  # on the diagonals
    B = O.Boxes3(b, bounds)
    d_o, k_o = B.nearest(p)
    with frw.Layout3.from_boxes(b, bounds) as L:
        assert L.info.max_list == k**3
        d, near = L.query(p)
        got = L.walk_trace(k, 0, 1500, 9)
    assert np.array_equal(d, d_o) and np.array_equal(near, k_o)
    for x, y in zip(got, B.walks(B.cfg(target=k, offset=1.0, seed=9), 0, 1500)):
        assert np.array_equal(x, y)


def test_lists_past_the_l2():
    """A layout whose lists are read from HBM takes the kernel that keeps the best
    entry in registers: nearest boxes, ties of lined-up boxes included, equal the
    oracle's."""
    b = frw.generate_layout3(3, 150_000, 20.0 * 150_000**0.5, 400.0, 5, 50, 5, 20, 2)
    B = O.Boxes3(b, grid=True)
    rng = np.random.default_rng(0)
    p = B.bounds[:3] + rng.random((60_000, 3)) * (B.bounds[3:] - B.bounds[:3])
    p[:20_000] = np.round(p[:20_000])
    p[20_000:30_000] = b[rng.integers(0, len(b), 10_000), 3:]
    with frw.Layout3.from_boxes(b) as L:
        assert L.info.list_entries * 32 > 256 << 20
        d, near = L.query(p)
    d_o, k_o = B.nearest(p)
    assert np.array_equal(d, d_o) and np.array_equal(near, k_o)
