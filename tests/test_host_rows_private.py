"""Result rows belong to one process and to one column: what a forked child
writes stays the child's, on both sides of the size from which the rows are
demand-zero pages, and a column kept alone keeps no other column's pages."""
import os
import subprocess
import sys

import pytest

import frw

FORK = """
import os, sys
sys.path.insert(0, sys.argv[1])
import frw
rows = frw._row_arrays(int(sys.argv[2]))
for r in rows:
    r[:] = 1
pid = os.fork()
if pid == 0:
    for r in rows:
        r[:] = 7
    os._exit(0)
assert os.waitpid(pid, 0)[1] == 0
assert all((r == 1).all() for r in rows), "the child's rows are the parent's"
"""


@pytest.mark.parametrize("cap", [64, (1 << 15) - 1, 1 << 15, 1_000_003])
def test_rows_are_not_shared_with_a_forked_child(cap):
    subprocess.run([sys.executable, "-c", FORK, os.path.dirname(os.path.dirname(frw.__file__)), str(cap)], check=True)


def test_columns_do_not_share_their_pages():
    owners = [getattr(r.base, "obj", r.base) for r in frw._row_arrays(1 << 15)]
    assert len({id(o) for o in owners}) == len(owners)
