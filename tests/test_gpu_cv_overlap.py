"""Control-variate training launches its steps so that a step's set-up overlaps
the update before it.  The parameters are those of the same steps run one launch
at a time (a child process in which every launch is waited for), bit for bit:
one CTA and several, a ragged last batch, many short steps."""
import os
import subprocess
import sys

import numpy as np
import pytest

import frw

TRAIN = """
import sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import frw
walks, batch, epochs = (int(v) for v in sys.argv[2:5])
with frw.Layout.from_rects(frw.generate_layout(11, 2000, 4472.0)) as L:
    cv = frw.ControlVariate(L, 7, frw.capacitance_opts(1.0, start_grid=256),
                            frw.cv_opts(train_walks=walks, batch=batch, epochs=epochs))
    np.save(sys.argv[5], cv.params())
    cv.close()
"""


@pytest.mark.gpu
@pytest.mark.parametrize("walks,batch,epochs", [(20_000, 64, 1), (50_000, 1024, 4), (100_001, 8192, 6),
                                                (200_000, 65_536, 8)])
def test_overlapped_steps_are_the_steps(tmp_path, walks, batch, epochs):
    out = []
    for blocking in ("0", "1"):
        f = str(tmp_path / f"{blocking}.npy")
        subprocess.run([sys.executable, "-c", TRAIN, os.path.dirname(os.path.dirname(frw.__file__)), str(walks),
                        str(batch), str(epochs), f], check=True, env=dict(os.environ, CUDA_LAUNCH_BLOCKING=blocking))
        out.append(np.load(f))
    assert np.isfinite(out[0]).all() and np.array_equal(out[0].view(np.uint32), out[1].view(np.uint32))
