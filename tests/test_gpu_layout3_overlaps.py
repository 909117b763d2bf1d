"""The overlap that a refused 3-D layout names is its lowest pair, whatever order
the device met the pairs in: one box over many, many pairs, all boxes equal."""
import numpy as np
import pytest

import frw

pytestmark = pytest.mark.gpu


def refused(b):
    with pytest.raises(frw.FrwError) as e:
        frw.Layout3.from_boxes(b)
    assert e.value.status == frw.E_ARG
    return str(e.value)


def lowest_pair(b):
    for i in range(len(b)):
        o = (b[i, :3] < b[i + 1:, 3:]).all(1) & (b[i + 1:, :3] < b[i, 3:]).all(1)
        if o.any():
            return f"boxes {i} and {i + 1 + int(np.argmax(o))} overlap"


@pytest.mark.parametrize("where", [0, 40, 998])
def test_one_box_over_many(where):
    """A slab over a third of the layout, whatever its index."""
    b = frw.generate_layout3(3, 999, 700.0, 400.0, 5, 50, 5, 20, 2)
    b[where] = [100, 100, 50, 500, 500, 350]
    names = {refused(b) for _ in range(6)}
    assert len(names) == 1 and lowest_pair(b) in names.pop()


@pytest.mark.parametrize("seed", [0, 1, 2])
def test_many_pairs(seed):
    rng = np.random.default_rng(seed)
    b = frw.generate_layout3(5, 5000, 1500.0, 400.0, 5, 50, 5, 20, 2)
    b[rng.integers(0, len(b), 700)] += np.float32(30)
    names = {refused(b) for _ in range(6)}
    assert len(names) == 1 and lowest_pair(b) in names.pop()


@pytest.mark.parametrize("n", [2, 33, 300_000])
def test_all_equal(n):
    assert "boxes 0 and 1 overlap" in refused(np.repeat(np.array([[0, 0, 0, 2, 2, 2]], np.float32), n, 0))
