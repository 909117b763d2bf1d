"""A matrix of targets with more nonzero rows than are brought in one piece, in a
pool with little more memory than its dense rows take: every target's row equals
that of its own run."""
import os
import subprocess
import sys

import pytest

import frw

RUN = """
import sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import frw
from cuda.bindings import runtime as rt

n, walks = 3000, 60_000
frw.device_check(0)
props = rt.cudaMemPoolProps()
props.allocType = rt.cudaMemAllocationType.cudaMemAllocationTypePinned
props.location.type = rt.cudaMemLocationType.cudaMemLocationTypeDevice
props.location.id = 0
props.maxSize = n * n * 24 + (64 << 20)
err, pool = rt.cudaMemPoolCreate(props)
assert int(err) == 0 and int(rt.cudaDeviceSetMemPool(0, pool)[0]) == 0
with frw.Layout3.from_boxes(frw.generate_layout3(5, n, 1096.0, 400.0, 5, 50, 5, 20, 2)) as L:
    rs = L.walk_batch(np.arange(n), walks, 5, frw.opts3(), capacity=1000)
    assert sum(len(r.conductor) for r in rs) > 1 << 18
    for t in (0, 1, 87, 1500, n - 1):
        one = L.walk(t, walks, 5)
        assert np.array_equal(rs[t].conductor, one.conductor) and np.array_equal(rs[t].hits, one.hits)
        assert rs[t].hops_total == one.hops_total and rs[t].escaped == one.escaped
        assert np.allclose(rs[t].sum_w, one.sum_w, rtol=1e-11, atol=1e-11 * np.abs(one.sum_w).sum())
assert all((np.diff(r.conductor) > 0).all() for r in rs)
"""


@pytest.mark.gpu
def test_more_rows_than_one_piece():
    pytest.importorskip("cuda.bindings.runtime")
    r = subprocess.run([sys.executable, "-c", RUN, os.path.dirname(os.path.dirname(frw.__file__))], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr[-2000:]
