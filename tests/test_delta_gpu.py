"""The per-fly delta update (fb_delta_apply) against the rule spelled out in float32."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.mark.parametrize("n_sel,batch,slots", [(1, 1, 1), (255, 5, 2), (257, 19, 3), (5000, 9, 9), (700, 33, 1)])
def test_delta_apply_orders_flies_and_synapses(torch, n_sel, batch, slots):
    """fb_delta_apply over runs of flies and blocks of synapses that do not divide evenly, bit for bit against
    the rule spelled out in float32 (slot order within a fly, non-learning slots left out)."""
    import scipy.sparse as sp

    from flyzero_b200 import _lib
    from flyzero_b200.gpu import BatchBrain

    rng = np.random.default_rng(n_sel)
    w = sp.random(n_sel + 40, n_sel + 40, density=2.0 * (n_sel + 40) / (n_sel + 40) ** 2, random_state=1, format="csr")
    w.data = rng.integers(1, 9, w.nnz) * rng.choice([1.0, -1.0], w.nnz)
    pos = np.sort(rng.choice(w.nnz, min(w.nnz, n_sel + 20), replace=False))
    gb = BatchBrain(w.astype(np.float32), batch=batch, plastic_pos=pos)
    sel = np.sort(rng.choice(len(pos), n_sel, replace=False)).astype(np.int32)
    n_tr, n_x = 37, 11
    pre, post = np.sort(rng.integers(0, n_tr, n_sel)).astype(np.int32), rng.integers(0, n_x, n_sel).astype(np.int32)
    trace, x = rng.random((batch, n_tr), np.float32), rng.standard_normal((batch, n_x)).astype(np.float32)
    coef = (rng.random(batch) * (rng.random(batch) < 0.8)).astype(np.float32)
    fly = np.arange(batch) // slots
    ptr = np.r_[0, np.cumsum(np.bincount(fly))].astype(np.int32)
    sign, wmax = np.sign(gb.w0).astype(np.float32), (np.float32(1.5) * np.abs(gb.w0)).astype(np.float32)
    want = gb.pw.cpu().numpy().copy()
    for f in range(len(ptr) - 1):
        d = np.zeros(n_sel, np.float32)
        for b in range(ptr[f], ptr[f + 1]):
            if coef[b] != 0:
                d = d + (coef[b] * trace[b, pre]) * x[b, post]
        for b in range(ptr[f], ptr[f + 1]):
            moved = sign[sel] * np.minimum(np.maximum(sign[sel] * (want[b, sel] + d), np.float32(0)), wmax[sel])
            want[b, sel] = np.where(d == 0, want[b, sel], moved)
    dev = [torch.as_tensor(a, device="cuda") for a in (sel, pre, post, trace, x, coef, ptr, np.arange(batch, dtype=np.int32), sign, wmax)]
    p = [C.c_void_p(t.data_ptr()) for t in dev]
    _lib.check(gb._L.fb_delta_apply(gb._h, p[0], p[1], p[2], n_sel, p[3], n_tr, p[4], n_x, p[5], p[6], p[7], len(ptr) - 1, p[8],
                                    p[9], None))
    torch.cuda.synchronize()
    np.testing.assert_array_equal(gb.pw.cpu().numpy(), want)
