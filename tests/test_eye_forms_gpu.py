"""The eye's default form (a grid kernel and a neuron kernel) against the four grid-wide kernels, bit for bit:
frames whose width is no multiple of a cell or of four, unaligned frames, every neuron of one kind, more
neurons than one chunk of a block, more instances than SMs, neurons out of range, no sustained or no
chromatic channels."""

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


@pytest.mark.parametrize("B,shape,cell,cells,kw", [
    (1, (224, 256), 4, 12_246, dict(transient_gain=4.0, sustained_gain=4.0, chromatic_gain=1.0)),
    (3, (61, 67), 4, 1025, dict(transient_gain=4.0, sustained_gain=4.0)),
    (2, (50, 64), 3, 31, dict(chromatic_gain=1.0)),
    (160, (32, 40), 4, 9000, dict(transient_gain=4.0, sustained_gain=4.0, chromatic_gain=1.0)),
    (5, (40, 36), 8, 4097, dict(sustained_gain=2.0)),
    (4, (33, 48), 1, 500, dict(transient_gain=1.0, sustained_gain=4.0, surround=7, shift=2)),
], ids=["fleet", "odd_width", "cell3", "many_instances", "cell8", "cell1"])
def test_default_form_equals_split_kernels(torch, B, shape, cell, cells, kw):
    from flyzero_b200.brain import LIFParams
    from flyzero_b200.gpu import BatchBrain
    from flyzero_b200.vision import BatchMotionEye, EyeLayout, MotionParams

    rng = np.random.default_rng(cells)
    h, w = shape
    gh, gw = h // cell, w // cell
    n = max(cells, 64)
    chan = rng.integers(0, 14, cells).astype(np.uint8)
    if cells == 31:
        chan[:] = 13                                               # every neuron of one kind
    gx, gy = rng.integers(0, gw, cells), rng.integers(0, gh, cells)
    gx[::17] = gw - 1
    gy[5::19] = gh - 1
    gx[3::101] = gw + 2                                            # out of range: skipped
    lo = EyeLayout(np.arange(cells), gx * cell, gy * cell, np.array(["left"] * cells), chan, gx, gy, rng.random(cells) < 0.9)
    p = MotionParams(gain=500.0, cell=cell, **kw)
    outs = []
    for kernels in ("auto", "split"):
        gb = BatchBrain(sp.csr_matrix((n, n), dtype=np.float32), LIFParams(), batch=B)
        eye = BatchMotionEye(gb, None, shape, p, eye_layout=lo, kernels=kernels)
        got = []
        r = np.random.default_rng(3)
        buf = torch.empty(B * h * w * 3 + 1, dtype=torch.uint8, device="cuda")
        for t in range(4):
            frames = torch.as_tensor(r.integers(0, 256, (B, h, w, 3), dtype=np.uint8))
            view = buf[t % 2:t % 2 + frames.numel()].view(B, h, w, 3)   # every second frame batch at an odd address
            view.copy_(frames)
            if t == 2:
                eye.reset([B - 1])
            eye.see(view, flip=r.random(B) < 0.5)
            got.append((eye.rates_dev.cpu().numpy().copy(), gb.p_ext.cpu().numpy().copy()))
        assert not eye.restart.any()
        outs.append(got)
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a[0].view(np.uint32), b[0].view(np.uint32))
        np.testing.assert_array_equal(a[1].view(np.uint32), b[1].view(np.uint32))
    assert outs[0][-1][0].max() > 0
