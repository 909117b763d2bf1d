"""3-D layout creation on the device: the checks (coordinates, empty boxes,
overlaps, touching faces) and the cell lists at the edges of their format --
grids smaller than a brick of cells, lists longer than a warp orders in shared
memory, candidates past what it holds, a second pass for the list buffer."""
import numpy as np
import pytest

import frw
import oracle as O

pytestmark = pytest.mark.gpu


def grid_boxes(k, pitch=3.0, edge=2.0, at=0.0):
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3) * pitch + at
    return np.concatenate([g, g + edge], 1).astype(np.float32)


def check(b, bounds=None, cells_per_box=0.0, n=6000, seed=0):
    B = O.Boxes3(b, bounds, grid=len(b) > 2000)
    rng = np.random.default_rng(seed)
    p = B.bounds[:3] + rng.random((n, 3)) * (B.bounds[3:] - B.bounds[:3])
    i = rng.integers(0, len(b), n // 2)
    p[: n // 2] = np.clip(b[i, :3] + rng.uniform(-2, 4, (n // 2, 3)), B.bounds[:3], B.bounds[3:])
    with frw.Layout3.from_boxes(b, bounds, cells_per_box) as L:
        d, k = L.query(p)
        info = L.info
    d_o, k_o = B.nearest(p)
    assert np.array_equal(d, d_o) and np.array_equal(k, k_o)
    return info


@pytest.mark.parametrize("n", [1, 2, 3, 5, 31, 33, 257])
@pytest.mark.parametrize("cells_per_box", [0.01, 1.0, 8.0, 300.0])
def test_small_grids(n, cells_per_box):
    b = frw.generate_layout3(n, n, 60.0 + 30.0 * n**0.5, 120.0, 5, 20, 5, 20, 2)
    check(b, cells_per_box=cells_per_box)


def test_long_lists_and_many_candidates():
    """A block of 4096 boxes: few coarse cells (hundreds of candidates a cell,
    past what a warp keeps and orders in shared memory), then in wide bounds,
    where distant cells of coarser levels face all of it."""
    b = grid_boxes(16)
    info = check(b, cells_per_box=0.01)
    assert info.max_list > 256
    info = check(b, cells_per_box=0.2)
    assert info.max_list > 40
    info = check(b, np.array([-900.0, -900, -900, 900, 900, 900]), seed=2)
    assert info.levels > 1


def test_lists_past_the_first_buffer():
    b = grid_boxes(12, pitch=2.5, edge=2.0)
    info = check(b, cells_per_box=1.0)
    assert info.list_entries > 9 * np.prod(info.grid[:]) + 4096


@pytest.mark.parametrize("where", [0, 1, 500, 998])
def test_overlaps_and_bad_boxes_are_found(where):
    b = frw.generate_layout3(3, 999, 700.0, 400.0, 5, 50, 5, 20, 2)
    for name, i, v in (("not finite", 3, np.nan), ("not finite", 0, -np.inf), ("not finite", 5, 2.0**24), ("empty", 3, b[where, 0])):
        c = b.copy()
        c[where, i] = v
        with pytest.raises(frw.FrwError) as e:
            frw.Layout3.from_boxes(c)
        assert e.value.status == frw.E_ARG and name in str(e.value) and f"box {where}:" in str(e.value)
    inside = b[where].copy()  # a box wholly inside another
    inside[:3] += 1
    inside[3:] -= 1
    with pytest.raises(frw.FrwError) as e:
        frw.Layout3.from_boxes(np.vstack([b, inside]))
    assert e.value.status == frw.E_ARG and f"boxes {where} and 999 overlap" in str(e.value)


def test_equal_boxes_are_refused_quickly_and_walls_accepted():
    same = np.repeat(grid_boxes(1), 20_000, 0)
    with pytest.raises(frw.FrwError) as e:
        frw.Layout3.from_boxes(same)
    assert "overlap" in str(e.value)
    # a floor under every box, touching them: one box over many bins
    b = grid_boxes(8)
    floor = np.array([[-5, -5, -4, 40, 40, 0]], np.float32)
    check(np.vstack([b, floor]))
