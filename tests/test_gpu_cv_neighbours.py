"""The list of a target's neighbours: targets with more neighbours than a list
holds at every reach, at the larger ones or at none, over more cells than are
looked at, with cells left to the tree, and without cells.  Features equal the
oracle's."""
import numpy as np
import pytest

import frw
import oracle as O

pytestmark = pytest.mark.gpu


def with_plate(n, w, h):
    """A uniform layout with a plate in its middle, rect 0."""
    r = frw.generate_layout(9, n, 100.0 * n**0.5).astype(float)
    c = 50.0 * n**0.5
    q = np.array([c - w / 2, c - h / 2, c + w / 2, c + h / 2]).round()
    keep = ~((r[:, 0] <= q[2]) & (r[:, 2] >= q[0]) & (r[:, 1] <= q[3]) & (r[:, 3] >= q[1]))
    return np.vstack([q[None], r[keep]])


def overlapping(n, size):
    rng = np.random.default_rng(2)
    a = rng.uniform(0, 100.0 * n**0.5, (n, 2)).round()
    return np.concatenate([a, a + rng.uniform(size / 2, size, (n, 2)).round()], 1)


# (a point inside several rects takes the deepest from cell lists, the first found from the tree)
@pytest.mark.parametrize("kind,cells", [(k, c) for k in ("point", "wire", "plate", "sheet", "overlapping")
                                        for c in (None, (0.0, 32), (2.0, 32), (16.0, 3))
                                        if k != "overlapping" or c in (None, (2.0, 32))])
def test_features_around_targets(kind, cells):
    r = {"point": with_plate(900, 8, 8), "wire": with_plate(2500, 3500, 6), "plate": with_plate(2500, 1500, 1500),
         "sheet": with_plate(6000, 5000, 5000), "overlapping": overlapping(900, 250.0)}[kind]
    rng = np.random.default_rng(1)
    t = r[0]
    with frw.Layout.from_rects(r) as L:
        if cells:
            L.set_cells(*cells)
        b = L.bounds
        p = np.concatenate([rng.uniform(t[:2] - 12, t[2:] + 12, (16_500, 2)), rng.uniform(t[:2] - 250, t[2:] + 250, (16_500, 2)),
                            np.round(rng.uniform(t[:2] - 30, t[2:] + 30, (500, 2)))]).clip(b[:2], b[2:])
        rec = np.zeros((len(p), 4))
        rec[:, :2] = p
        rec[:, 2] = rng.choice([1.0, 2.5, 7.0], len(p))
        got = L.cv_features(0, rec)
        few = L.cv_features(0, rec[:1000])  # without the list
    assert np.array_equal(got[:1000], few)
    assert np.array_equal(got, O.cv_features(r, 0, rec))
