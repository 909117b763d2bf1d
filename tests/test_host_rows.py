"""Result rows of the Python mirror: writable zeros of the asked length on both
sides of the size from which they are demand-zero pages."""
import numpy as np
import pytest

import frw


@pytest.mark.parametrize("cap", [0, 1, 64, (1 << 15) - 1, 1 << 15, 1_000_003])
def test_row_arrays(cap):
    rows = frw._row_arrays(cap)
    assert [r.dtype for r in rows] == [np.int64, np.uint64] + [np.float64] * 4
    for k, r in enumerate(rows):
        assert r.shape == (cap,) and not r.any() and r.flags.writeable
        r[-3:] = k + 1  # no two overlap
    for k, r in enumerate(rows):
        assert (r[-3:] == k + 1).all() and not r[:-3].any()
        assert r[: cap // 2].base is r  # a result's front keeps the whole row


@pytest.mark.gpu
@pytest.mark.parametrize("walks", [1, 500_000, 700_000, 1_500_001])
def test_trace_copies_at_every_size(walks):
    """Per-walk records through one copy and (past 16 MiB) through the copying
    threads: the counts of the same walks' rows."""
    with frw.Layout.from_rects(frw.generate_layout(3, 500, 2236.0)) as L:
        end, hops, b1, w = L.walk_trace(2, 0, walks, 5, frw.capacitance_opts(1.0))
        r = L.walk(2, walks, 5, frw.capacitance_opts(1.0))
        again = L.walk_trace(2, 0, walks, 5, frw.capacitance_opts(1.0))
    assert r.hops_total == int(hops.sum()) and r.escaped == int((end == -1).sum())
    k, n = np.unique(end[end >= 0], return_counts=True)
    assert np.array_equal(r.conductor, k) and np.array_equal(r.hits, n)
    assert ((b1 >= -1) & (b1 < 200)).all() and np.isfinite(w).all()
    assert all(np.array_equal(x, y) for x, y in zip(again, (end, hops, b1, w)))
