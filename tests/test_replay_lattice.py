"""The expand-and-bisect square from the clearance alone (the closed form of
the replay's decisions, csrc/query.cuh) against the oracle's loop, over
layouts from under 2 units wide (no halving) to 2^24 (23 halvings)."""
import numpy as np
import pytest

import frw
import oracle as O

# bounds x0, y0, x1, y1 and the number of rects
BOUNDS = [(0, 0, 1.25, 1), (0, 0, 1.9375, 1.5), (0, 0, 3, 2.5), (-7, 3, 33, 21), (0, 0, 1020, 1020), (0, 0, 10198, 9000),
          (-51000, -51000, 51000, 50990), (8388000, 8388000, 8388600, 8388400), (-2.0**23, -2.0**23, 2.0**23 - 8, 2.0**23 - 8)]


def layout(bounds):
    rng = np.random.default_rng(5)
    b = np.asarray(bounds, dtype=np.float64)
    w = b[2:] - b[:2]
    k = 40
    lo = b[:2] + w * rng.uniform(0.02, 0.9, (k, 2))
    r = np.concatenate([lo, lo + w * rng.uniform(0.001, 0.06, (k, 2))], 1)
    if w.max() > 100:
        r = np.round(r)  # integer corners: ties with integer points
    r = r.astype(np.float32).astype(np.float64)
    r[:, 2:] = np.minimum(r[:, 2:], b[2:])
    p = np.stack([rng.uniform(b[0], b[2], 4000), rng.uniform(b[1], b[3], 4000)], 1)
    p[:600] = np.round(p[:600])  # may lie on rects and on the bounds
    near = rng.integers(0, k, 1500)  # distances around the first boxes p +- 1 and p +- 2
    p[600:2100, 0] = r[near, 0] - rng.choice([0.5, 1, 1 + 1e-9, 1.75, 2, 2 - 1e-9, 2.25, 3], 1500)
    p[600:2100, 1] = rng.uniform(r[near, 1], r[near, 3])
    return r, b, p


def closed_form(r, b, p):
    """(squares, settled): the device rule in numpy; settled where the
    clearance decides every box."""
    x, y = p[:, 0], p[:, 1]
    d = np.minimum(np.minimum(x - b[0], b[2] - x), np.minimum(y - b[1], b[3] - y))
    outside = d < 0
    gx = np.maximum(r[None, :, 0] - x[:, None], x[:, None] - r[None, :, 2])
    gy = np.maximum(r[None, :, 1] - y[:, None], y[:, None] - r[None, :, 3])
    d = np.where(outside, -1.0, np.minimum(d, np.maximum(gx, gy).min(1)))
    w = (b[2:] - b[:2]).max()
    dist = 0.05 * w
    K = 0
    while dist * 0.5**K > np.float32(0.095):
        K += 1
    delta = (4.0 * max(np.abs(b).max(), w) + 16.0) * 2.0**-39  # twice the library's window
    scale = 2.0**K / dist
    one = d < 1.5
    h = np.where(one, 1.0, 2.0)
    e = d - h
    first = e < -delta
    tie = np.abs(e) <= delta
    t = (d - 1.0) * scale
    q = np.floor(np.maximum(t, 0)).astype(np.int64)
    guard = 2 * delta * scale + 20 * 2.0**(K - 50)
    lattice = ~first & ~one
    settled = first | (one & ~tie) | (lattice & ~tie & (t - q > guard) & (t - q < 1 - guard) & (1 <= K <= 26))
    o = np.where((first & one)[:, None] | lattice[:, None], np.array([-1.0, -1, 1, 1]), np.array([-2.0, -2, 2, 2])) + p[:, [0, 1, 0, 1]]
    s = np.array([-1.0, -1, 1, 1])
    go = lattice & settled
    grown = q >> K
    for k in range(0, (grown[go].max() + 1) if go.any() else 0):
        o = np.where((go & (k <= grown))[:, None], o + s * dist, o)
    step = dist
    for k in range(1, K + 1):
        step *= 0.5
        grow = (q >> (K - k + 1)) & 1 if k > 1 else np.zeros_like(q)
        o = np.where(go[:, None], o + s * np.where(grow == 1, step, -step)[:, None], o)
    return np.where((go & ((q & 1) == 0))[:, None], o - s * step, o), settled


@pytest.mark.parametrize("bounds", BOUNDS)
def test_closed_form_equals_the_loop(bounds):
    r, b, p = layout(bounds)
    sq, settled = closed_form(r, b, p)
    ref, _ = O.Grid(r, b).query_batch(p)
    assert np.array_equal(sq[settled], ref[settled])
    if (b[2:] - b[:2]).max() > 3:  # the rule is not a corner case: it decides nearly every generic point
        assert settled[2100:].mean() > 0.95


@pytest.mark.gpu
@pytest.mark.parametrize("bounds", BOUNDS)
def test_device_squares(bounds):
    r, b, p = layout(bounds)
    ref, hit_ref = O.Grid(r, b).query_batch(p)
    far = np.array([[np.nan, b[1] + 1], [b[0] + 1, np.nan], [np.inf, 0], [0, -np.inf], [b[0] - 5, b[1]], [b[2], b[3] + 700]])
    with frw.Layout.from_rects(r, b) as L:
        for cells in (True, False):
            if not cells:
                L.set_cells(0)
            sq, hit = L.query(p)
            assert np.array_equal(sq, ref) and np.array_equal(hit, hit_ref)
            sq, hit = L.query(far)  # outside the bounds: the first box, no rect
            assert np.array_equal(sq, far[:, [0, 1, 0, 1]] + np.array([-1.0, -1, 1, 1]), equal_nan=True)
            assert (hit == -1).all()
