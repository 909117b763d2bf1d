"""3-D grids are built in the memory that their lists need: in a pool too small
for the room the build would like to have first, and for a second copy of the
lists, the layout is the one built without a limit."""
import os
import subprocess
import sys

import pytest

import frw

LIMITED = """
import sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import frw
from cuda.bindings import runtime as rt

def build():
    b = frw.generate_layout3(5, 64, 160.0, 400.0, 5, 50, 5, 20, 2)
    with frw.Layout3.from_boxes(b, None, 10_000.0) as L:
        p = L.bounds[:3] + np.random.default_rng(0).random((20_000, 3)) * (L.bounds[3:] - L.bounds[:3])
        return L.info, L.query(p), L.walk_trace(3, 0, 2000, 5)

free = build()
assert 32 * (10 * np.prod(free[0].grid[:]) + 4096) > 2 * int(sys.argv[2]) > 8 * 32 * free[0].list_entries
props = rt.cudaMemPoolProps()
props.allocType = rt.cudaMemAllocationType.cudaMemAllocationTypePinned
props.location.type = rt.cudaMemLocationType.cudaMemLocationTypeDevice
props.location.id = 0
props.maxSize = int(sys.argv[2])
err, pool = rt.cudaMemPoolCreate(props)
assert int(err) == 0
assert int(rt.cudaDeviceSetMemPool(0, pool)[0]) == 0
small = build()
assert small[0].list_entries == free[0].list_entries and small[0].max_list == free[0].max_list
for a, b in zip(small[1] + small[2], free[1] + free[2]):
    assert np.array_equal(a, b)
"""


@pytest.mark.gpu
def test_grid_in_a_small_pool():
    pytest.importorskip("cuda.bindings.runtime")
    r = subprocess.run([sys.executable, "-c", LIMITED, os.path.dirname(os.path.dirname(frw.__file__)), str(96 << 20)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
