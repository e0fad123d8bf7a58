"""Eye grids at the limit of a block's shared memory: the largest that the two-kernel form takes, and the ones
just beyond it, which the four grid-wide kernels take. Both against the four kernels, bit for bit. (Grids whose
tables alone come to exactly the limit were refused when the kernel had 16 static bytes beside them.)"""

import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("gh,gw,kw", [
    (128, 130, {}), (130, 128, {}), (104, 160, {}),                                 # motion: 3 floats a cell, 58,112 in all
    (151, 110, {}), (151, 111, {}),
    (96, 104, dict(chromatic_gain=1.0)), (78, 128, dict(chromatic_gain=1.0)),       # colours: 5 floats a cell
    (78, 90, dict(sustained_gain=2.0, chromatic_gain=1.0)),                          # all: 6 and the integral image
    (79, 90, dict(sustained_gain=2.0, chromatic_gain=1.0)),
], ids=lambda v: str(v) if isinstance(v, int) else "+".join(v) or "motion")
def test_grids_at_the_shared_memory_limit(torch, gh, gw, kw):
    from flyzero_b200.brain import LIFParams
    from flyzero_b200.gpu import BatchBrain
    from flyzero_b200.vision import BatchMotionEye, EyeLayout, MotionParams

    B, cells, cell = 2, 700, 2
    rng = np.random.default_rng(gh)
    chan = rng.integers(0, 14, cells).astype(np.uint8)
    gx, gy = rng.integers(0, gw, cells), rng.integers(0, gh, cells)
    lo = EyeLayout(np.arange(cells), gx * cell, gy * cell, np.array(["left"] * cells), chan, gx, gy, rng.random(cells) < 0.9)
    p = MotionParams(gain=500.0, cell=cell, **kw)
    outs = []
    for kernels in ("auto", "split"):
        gb = BatchBrain(sp.csr_matrix((cells, cells), dtype=np.float32), LIFParams(), batch=B)
        eye = BatchMotionEye(gb, None, (gh * cell, gw * cell), p, eye_layout=lo, kernels=kernels)
        r = np.random.default_rng(3)
        for _ in range(3):
            frames = torch.as_tensor(r.integers(0, 256, (B, gh * cell, gw * cell, 3), dtype=np.uint8)).cuda()
            eye.see(frames, flip=[False, True])
        assert not eye.restart.any()
        outs.append((eye.rates_dev.cpu().numpy().view(np.uint32), gb.p_ext.cpu().numpy().view(np.uint32)))
    np.testing.assert_array_equal(outs[0][0], outs[1][0])
    np.testing.assert_array_equal(outs[0][1], outs[1][1])
    assert outs[1][0].any()
