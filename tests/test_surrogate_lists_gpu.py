"""The surrogate's list kernels and conversions at the edges of their tiles, against plain PyTorch: FP32 -> bf16
with its transposed copy (vector and element form), Adam on several parameters at once, column sums of
several matrices at once, and the GEMM's row stores where rows are not 16-byte aligned."""

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


def _p(t):
    return None if t is None else C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("rows,cols,ldt,shift", [(1, 4, 4, 0), (63, 64, 64, 0), (65, 68, 72, 0), (130, 1280, 132, 0), (64, 10, 64, 0),
                                                 (65, 64, 67, 0), (66, 64, 68, 1)])
def test_to_bf16_with_transpose(torch, rows, cols, ldt, shift):
    from flyzero_b200 import _lib

    L = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows * cols + shift, device="cuda", generator=g)[shift:]
    out = torch.zeros(rows * cols, dtype=torch.bfloat16, device="cuda")
    out_t = torch.full((cols, ldt), 7.0, dtype=torch.bfloat16, device="cuda")
    for o in (out, None):
        out_t.fill_(7.0)
        _lib.check(L.fs_to_bf16(_p(x), rows * cols, _p(o), _p(out_t), rows, cols, ldt, None))
        want = x.to(torch.bfloat16).view(rows, cols)
        assert torch.equal(out.view(rows, cols), want)
        assert torch.equal(out_t[:, :rows], want.T) and bool((out_t[:, rows:] == 7.0).all())


def test_adam_list(torch):
    """Weights with transposed copies, vectors and runs across several rows of tiles, eight at once: weights and moments
    within a few roundings of the formula in float64, the copies exactly the weight's bf16."""
    from flyzero_b200 import _lib

    L = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(1)
    shapes = [(33, 70, True), (1, 1, False), (1, 1023, False), (1, 1024, False), (1, 1025, False), (1, 70_001, False), (10, 512, True),
              (64, 32, True)]
    lr, b1, b2, eps, t = *(float(np.float32(x)) for x in (1e-3, 0.9, 0.999, 1e-8)), 5      # (as the C ABI receives them)
    items, keep = [], []
    for r, c, tr in shapes:
        n = r * c
        w, gr, m = (torch.randn(n, device="cuda", generator=g) for _ in range(3))
        v = torch.rand(n, device="cuda", generator=g)
        wb = torch.zeros(n, dtype=torch.bfloat16, device="cuda")
        wt = torch.zeros((c, r + 3), dtype=torch.bfloat16, device="cuda") if tr else None
        keep.append((w, gr, m, v, wb, wt, [x.double().clone() for x in (w, gr, m, v)], r, c))
        items.append(_lib.AdamItem(*(x.data_ptr() if x is not None else None for x in (w, gr, m, v, wb, wt)), n, r, c, r + 3))
    _lib.check(L.fs_adam_list((_lib.AdamItem * 8)(*items), 8, lr, b1, b2, eps, t, None))
    for w, gr, m, v, wb, wt, (w0, g0, m0, v0), r, c in keep:
        mm, vv = b1 * m0 + (1 - b1) * g0, b2 * v0 + (1 - b2) * g0 * g0
        want = w0 - lr * (mm / (1 - b1 ** t)) / ((vv / (1 - b2 ** t)).sqrt() + eps)
        # float32: b2 carries 6e-8 of itself, which c2 = 1 - b2^t divides by 0.005 (6e-5 of the update's square, so
        # 3e-5 of the update); the weight is rounded twice (1.2e-7)
        assert float(((m - mm).abs() / (mm.abs() + 0.1)).max()) < 1e-6
        assert float(((v - vv).abs() / vv).max()) < 1e-6
        assert float(((w - want).abs() / (1.2e-7 * want.abs() + 1e-4 * (want - w0).abs() + 1e-9)).max()) < 1.0
        assert torch.equal(wb, w.to(torch.bfloat16))
        if wt is not None:
            assert torch.equal(wt[:, :r], w.view(r, c).T.to(torch.bfloat16)) and bool((wt[:, r:] == 0).all())
    assert L.fs_adam_list((_lib.AdamItem * 8)(*items), 9, lr, b1, b2, eps, t, None) == _lib.FB_ERR_ARG


@pytest.mark.parametrize("M", [1, 255, 513, 4096])
def test_colsum_list_equals_single_sums(torch, M):
    from flyzero_b200 import _lib

    L = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(M)
    xs = [torch.randn((M, ld), device="cuda", generator=g).to(torch.bfloat16) for ld in (512, 33, 16)]
    ns = (512, 33, 10)
    outs = [torch.empty(n, device="cuda") for n in ns]
    items = [_lib.ColsumItem(x.data_ptr(), o.data_ptr(), n, x.shape[1]) for x, o, n in zip(xs, outs, ns)]
    _lib.check(L.fs_colsum_list((_lib.ColsumItem * 3)(*items), 3, M, None))
    for x, o, n in zip(xs, outs, ns):
        one = torch.empty(n, device="cuda")
        _lib.check(L.fs_colsum(_p(x), M, n, x.shape[1], _p(one), None))
        assert torch.equal(o, one)
        torch.testing.assert_close(o.double(), x[:, :n].double().sum(0), rtol=1e-5, atol=1e-6 * M)


@pytest.mark.parametrize("M,N,K,ldo,shift", [(129, 64, 64, 65, 0), (64, 80, 128, 80, 1), (200, 48, 1024, 52, 0), (130, 70, 2048, 72, 0)])
def test_gemm_rows_that_do_not_start_on_16_bytes(torch, M, N, K, ldo, shift):
    """The row-store epilogue falls back element by element; both forms agree with FP32 sums of the same operands."""
    from flyzero_b200 import _lib

    L = _lib.load()
    g = torch.Generator(device="cuda").manual_seed(M)
    A = torch.randn((M, K), device="cuda", generator=g).to(torch.bfloat16)
    B = torch.randn((N, K), device="cuda", generator=g).to(torch.bfloat16)
    bias = torch.randn(N, device="cuda", generator=g)
    ref = A.float() @ B.float().T
    out = torch.full((M * ldo + shift,), 5.0, device="cuda")
    view = out[shift:].view(M, ldo)
    _lib.check(L.fs_gemm(_p(A), _p(B), M, N, K, K, K, 2, _p(bias), None, _p(view), None, None, ldo, 0, None))
    torch.testing.assert_close(view[:, :N], ref + bias, rtol=2e-5 * K, atol=2e-5 * K)
    assert bool((view[:, N:] == 5.0).all())
    z = torch.empty((M, ldo), device="cuda")
    h = torch.full((M, ldo), 5.0, dtype=torch.bfloat16, device="cuda")
    ht = torch.empty((N, M), dtype=torch.bfloat16, device="cuda")
    _lib.check(L.fs_gemm(_p(A), _p(B), M, N, K, K, K, 1, _p(bias), None, _p(z), _p(h), _p(ht), ldo, M, None))
    torch.testing.assert_close(z[:, :N], ref + bias, rtol=2e-5 * K, atol=2e-5 * K)
    torch.testing.assert_close(h[:, :N].float(), torch.nn.functional.gelu(z[:, :N]), rtol=1e-2, atol=1e-2)
    assert torch.equal(ht.T, h[:, :N]) and bool((h[:, N:] == 5.0).all())
