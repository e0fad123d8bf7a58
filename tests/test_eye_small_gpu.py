"""The eye's one-launch form (a block per instance that takes its grid too), its half-sized blocks and its unsorted
neurons, each at sizes of more and of less than a block's chunk of neurons, against the four grid-wide
kernels bit for bit; and which calls take one launch."""

import numpy as np
import pytest
import scipy.sparse as sp

import test_eye_forms_gpu as forms
from test_eye_forms_gpu import torch  # noqa: F401

pytestmark = pytest.mark.gpu

ALL = dict(transient_gain=4.0, sustained_gain=4.0, chromatic_gain=1.0)


@pytest.mark.parametrize("B,shape,cell,cells,kw", [
    (1, (32, 32), 4, 300, ALL),                                 # one launch, less than a block of neurons
    (30, (61, 67), 4, 1000, ALL),
    (148, (50, 64), 3, 3287, ALL),                              # every SM an instance: sorted, cells of any size
    (148, (32, 40), 4, 9000, ALL),                              # ... three chunks
    (148, (32, 40), 4, 9000, {}),                               # ... unsorted
    (5, (80, 96), 4, 4099, dict(transient_gain=1.0, chromatic_gain=1.0)),   # two launches, unsorted
    (149, (32, 40), 4, 300, ALL),                               # half-sized blocks
    (149, (32, 40), 4, 9000, ALL),                              # ... two launches, five chunks
    (149, (33, 41), 2, 4097, dict(chromatic_gain=1.0)),
    (297, (32, 40), 4, 2500, ALL),                              # ... more than the SMs hold at once
], ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else "+".join(v) or "motion" if isinstance(v, dict) else str(v))
def test_small_forms_equal_split_kernels(torch, B, shape, cell, cells, kw):  # noqa: F811
    forms.test_default_form_equals_split_kernels(torch, B, shape, cell, cells, kw)


@pytest.mark.parametrize("B,gh,gw,cells,launches", [(1, 8, 8, 300, 1), (30, 16, 16, 1000, 1), (148, 25, 40, 3287, 1),
                                                    (1, 25, 40, 3287, 2), (64, 56, 64, 12_246, 2)])
def test_launches(torch, B, gh, gw, cells, launches):  # noqa: F811
    from flyzero_b200.brain import LIFParams
    from flyzero_b200.gpu import BatchBrain
    from flyzero_b200.vision import BatchMotionEye, EyeLayout, MotionParams

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the sizes are those of 148 SMs")
    rng = np.random.default_rng(cells)
    gx, gy = rng.integers(0, gw, cells), rng.integers(0, gh, cells)
    lo = EyeLayout(np.arange(cells), gx * 4, gy * 4, np.array(["left"] * cells), rng.integers(0, 14, cells).astype(np.uint8),
                   gx, gy, np.ones(cells, bool))
    gb = BatchBrain(sp.csr_matrix((cells, cells), dtype=np.float32), LIFParams(), batch=B)
    eye = BatchMotionEye(gb, None, (gh * 4, gw * 4), MotionParams(gain=500.0, **ALL), eye_layout=lo)
    before = gb.launches
    eye.see(torch.zeros((B, gh * 4, gw * 4, 3), dtype=torch.uint8, device="cuda"))
    assert gb.launches - before == launches
