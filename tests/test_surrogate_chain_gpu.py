"""The surrogate's kernels are launched as a chain in which the next kernel is set up while its predecessor runs. The
result must not depend on that: a captured and replayed step, a step behind other work in the
stream and a step whose operands the kernel just before has written give the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch(rows, dims, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    X = torch.randn((rows, dims[0]), device="cuda", generator=gen)
    return X, torch.poisson(torch.ones((rows, dims[-1]), device="cuda"), generator=gen)


def _step(net, X, Y):
    z = net.forward(X, training=True)
    loss = net.backward(Y)
    return z, loss, [t for pair in net.grads for t in pair]


@pytest.mark.parametrize("rows", [8, 40, 128, 704])
def test_chain_is_ordered(rows):
    from flyzero_b200.surrogate import DIMS, MLP
    one, two = MLP(seed=0), MLP(seed=0)
    X, Y = _batch(rows, DIMS, rows)
    z, loss, grads = _step(one, X, Y)
    z, loss, grads = z.clone(), loss.clone() if torch.is_tensor(loss) else loss, [t.clone() for t in grads]
    torch.cuda.synchronize()

    _step(two, X + 1, Y)                                 # buffers made, and full of other values
    torch.cuda.synchronize()
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    staged = torch.empty_like(X)
    with torch.cuda.stream(stream), torch.cuda.graph(graph, stream=stream):
        staged.copy_(X)                                  # an ordinary launch before the chain ...
        z2, loss2, grads2 = _step(two, staged, Y)
        read = z2 * 1.0                                  # ... and one behind it
    for _ in range(3):
        staged.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(read, z)
        assert float(loss2) == float(loss)
        assert all(torch.equal(p, q) for p, q in zip(grads, grads2))
