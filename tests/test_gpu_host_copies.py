"""Results at every size into memory that the driver writes to directly (page-
locked or device memory given as the host's), and into pageable memory, which
large ones reach through the copying threads: the same arrays."""
import ctypes as C

import numpy as np
import pytest

import frw

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def layout():
    with frw.Layout.from_rects(frw.generate_layout(3, 500, 2236.0)) as L:
        yield L


def query(L, p, sq, hit):
    return frw.lib().frw_query_batch(L._h, C.c_void_p(p.data_ptr()), C.c_int64(len(p)), C.c_void_p(sq.data_ptr()),
                                     C.c_void_p(hit.data_ptr()), frw.MEM_HOST, None)


@pytest.mark.parametrize("n", [1000, 419_430, 419_431, 1_500_001])
def test_page_locked_results(layout, n):
    import torch

    b = layout.bounds
    p = torch.rand((n, 2), dtype=torch.float64) * torch.tensor(b[2:] - b[:2]) + torch.tensor(b[:2])
    out = []
    for pinned in (False, True):
        sq = torch.empty((n, 4), dtype=torch.float64, pin_memory=pinned)
        hit = torch.empty(n, dtype=torch.int64, pin_memory=pinned)
        assert query(layout, p, sq, hit) == 0
        out.append((sq.numpy(), hit.numpy()))
    assert all(np.array_equal(x, y) for x, y in zip(*out))


@pytest.mark.parametrize("n", [1000, 1_500_001])
def test_device_memory_as_results(layout, n):
    import torch

    p = torch.rand((n, 2), dtype=torch.float64) * 2000.0
    out = []
    for device in ("cpu", "cuda"):
        sq = torch.empty((n, 4), dtype=torch.float64, device=device)
        hit = torch.empty(n, dtype=torch.int64, device=device)
        assert query(layout, p, sq, hit) == 0
        out.append((sq.cpu().numpy(), hit.cpu().numpy()))
    assert all(np.array_equal(x, y) for x, y in zip(*out))
