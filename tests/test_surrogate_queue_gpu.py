"""The surrogate's training steps queued one after the other, with nothing waiting between them, against the same
steps with the device synchronised after every kernel: weights, moments, gradients and outputs bit for bit.
Each kernel of the chain then reads what its predecessors wrote while it was already resident (the forward
pass the biases of the Adam update before it)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


class Synchronised:
    """The library with the device synchronised after every call."""

    def __init__(self, lib, torch):
        self._lib, self._torch = lib, torch

    def __getattr__(self, name):
        fn = getattr(self._lib, name)

        def call(*args):
            rc = fn(*args)
            self._torch.cuda.synchronize()
            return rc
        return call


@pytest.mark.parametrize("M", [8, 256, 1024])
def test_queued_steps_equal_synchronised_steps(torch, M):
    from flyzero_b200.surrogate import MLP

    rng = np.random.default_rng(M)
    data = [(torch.as_tensor(rng.standard_normal((M, 1280)).astype(np.float32), device="cuda"),
             torch.as_tensor(rng.poisson(2.0, (M, 10)).astype(np.float32), device="cuda")) for _ in range(6)]
    nets = [MLP(seed=1), MLP(seed=1)]
    nets[1].L = Synchronised(nets[1].L, torch)
    outs = []
    for net in nets:
        torch.cuda.synchronize()
        got = []
        for X, Y in data:
            net.train_step(X, Y)
            got.append(net.forward(X).clone())
        torch.cuda.synchronize()
        outs.append([*got, *net.W, *net.b, *(t for p in (*net.m, *net.v, *net.grads) for t in p)])
    for a, b in zip(*outs):
        assert torch.isfinite(a).all()
        np.testing.assert_array_equal(a.cpu().numpy().view(np.uint32), b.cpu().numpy().view(np.uint32))
