"""3-D walks from several host threads at once, each with its own landing table
and stream: long enough for the blocks that hold their table in shared memory,
whose size differs from thread to thread.  Every run gives the counts of the
same run alone."""
import threading

import numpy as np
import pytest

import frw


@pytest.mark.gpu
@pytest.mark.parametrize("tables", [(50, 20, 49, 21), (8, 64, 50, 65)])
def test_threads_with_different_tables(tables):
    import torch

    walks, runs = 160_000, 1200
    with frw.Layout3.from_boxes(frw.generate_layout3(7, 100, 200.0, 400.0, 5, 50, 5, 20, 2)) as L:
        alone = {n: L.walk(3, walks, 5, frw.opts3(nsample=n)) for n in tables}
        failed = []

        def run(n):
            stream = torch.cuda.Stream()
            try:
                for _ in range(runs):
                    r = L.walk(3, walks, 5, frw.opts3(nsample=n), stream=stream.cuda_stream)
                    if not np.array_equal(r.hits, alone[n].hits) or r.hops_total != alone[n].hops_total:
                        failed.append((n, "other counts"))
            except frw.FrwError as e:
                failed.append((n, str(e)))

        threads = [threading.Thread(target=run, args=(n,)) for n in tables]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert not failed, failed[:3]
