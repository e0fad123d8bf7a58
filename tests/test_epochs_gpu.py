"""The persistent engine's epochs at the sizes and options where they can go wrong, bit for bit against
the oracle: rows that end inside a tile or a quad, runs shorter than an epoch or not a multiple of one,
every epoch length from 1 (n_delay 3) to 6, instances that stop within an epoch, biased and plastic
quads, more spikes and more inputs per CTA than its buffers hold, and both engines in turn on one
simulation."""

import numpy as np
import pytest
import scipy.sparse as sp

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


def _net(n, degree, seed, integral):
    rng = np.random.default_rng(seed)
    rows = np.repeat(np.arange(n), degree)
    cols = rng.integers(0, n, n * degree)
    w = sp.coo_matrix((np.ones(n * degree), (rows, cols)), (n, n)).tocsr()
    w.sum_duplicates()
    size = rng.integers(1, 9, w.nnz) if integral else rng.uniform(0.3, 9.0, w.nnz)
    w.data = (size * rng.choice([1.0, 1.0, -1.0], w.nnz)).astype(np.float32)
    return w


def _pair(torch, n, B, delay, degree=8, integral=True, plastic=0.0, bias=0.0, driven=0.3, hz=150.0, seed=3):
    """The engine and the oracle on one network with the same drive."""
    from flyzero_b200.brain import LIFParams
    from flyzero_b200.gpu import BatchBrain

    rng = np.random.default_rng(seed)
    w = _net(n, min(degree, n), seed, integral)
    pos = np.sort(rng.choice(w.nnz, int(plastic * w.nnz), replace=False)) if plastic else None
    gb = BatchBrain(w, LIFParams(delay=delay), batch=B, seed=seed, plastic_pos=pos)
    eo = O.EngineOracle(w, O.Params(delay=delay), batch=B, plastic_pos=pos, seed=seed)
    gb.set_schedule("persistent")
    idx = np.sort(rng.choice(n, max(1, int(driven * n)), replace=False))
    rates = rng.uniform(0.0, 2.0 * hz, (B, len(idx))).astype(np.float32)
    gb.set_input(idx, rates)
    j = eo.slots(idx)
    eo.p_ext[:, j] = rates * np.float32(0.1 / 1000.0)
    if bias:
        at = rng.choice(n, max(1, int(bias * n)), replace=False)
        mv = rng.uniform(0.0, 6.0, (B, len(at))).astype(np.float32)
        gb.set_bias(at, mv)
        j = eo.slots(at)
        eo.bias_ext[:, j] = mv
        np.testing.assert_array_equal(gb.bias_ext.cpu().numpy(), eo.bias_ext)
    if pos is not None:
        gb.pw *= torch.as_tensor(rng.uniform(0.5, 2.0, gb.pw.shape).astype(np.float32), device=gb.device)
        eo.pw[:] = gb.pw.cpu().numpy()
    return gb, eo


def _same(gb, eo, c, want):
    np.testing.assert_array_equal(c.cpu().numpy(), want)
    for name in ("v", "g", "ref"):
        np.testing.assert_array_equal(getattr(gb, name).cpu().numpy(), getattr(eo, name))


@pytest.mark.parametrize("integral", [True, False], ids=["counts", "float"])
@pytest.mark.parametrize("n,B,delay", [(1, 1, 1.8), (3, 5, 1.8), (16, 2, 0.3), (127, 3, 0.5), (129, 2, 0.9), (1000, 7, 1.8),
                                       (5003, 13, 1.2), (30_011, 6, 1.8)])
def test_epochs_match_the_oracle(torch, n, B, delay, integral):
    gb, eo = _pair(torch, n, B, delay, integral=integral, plastic=0.05 if n > 3 else 0.0, bias=0.03)
    assert gb.info().epoch == max(1, min(6 if integral else 4, gb.n_delay // 3))
    for steps in (1, 2, 41, 7, 60):
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps))
    gb.check()


@pytest.mark.parametrize("plastic,bias", [(0.5, 0.0), (0.0, 0.9), (0.3, 0.4)])
def test_many_special_quads(torch, plastic, bias):
    gb, eo = _pair(torch, 3001, 9, 1.8, plastic=plastic, bias=bias)
    for steps in (30, 55):
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps))
    gb.check()


def test_more_spikes_and_inputs_than_the_buffers_hold(torch):
    # every neuron is an input that is kicked at once: all pairs of a CTA (2,163) fire in the first step
    gb, eo = _pair(torch, 40_000, 8, 1.8, degree=3, driven=1.0, hz=20_000.0)
    assert 8 * 40_000 / gb.info().ctas > 2048
    for steps in (9, 30):
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps))
    gb.check()


def test_instances_that_stop_within_an_epoch(torch):
    gb, eo = _pair(torch, 2001, 6, 1.8, plastic=0.05, bias=0.03)
    _same(gb, eo, gb.run_steps(20), eo.run_steps(20))
    left = np.array([0, 1, 5, 13, 40, -1])
    gb.set_run_length(left)
    stop = np.where(left < 0, 2 ** 62, eo.t + left).astype(np.int64)
    _same(gb, eo, gb.run_steps(37), eo.run_steps(37, stop_tick=stop))
    gb.reset([0, 2])
    eo.reset_flies([0, 2])
    live = [0, 2, 5]                                    # the others stay where they stopped
    gb.set_run_length(np.where(np.isin(np.arange(6), live), -1, 0))
    stop = np.where(np.isin(np.arange(6), live), 2 ** 62, eo.t).astype(np.int64)
    _same(gb, eo, gb.run_steps(31), eo.run_steps(31, stop_tick=stop))
    gb.check()


def test_engines_in_turn(torch):
    gb, eo = _pair(torch, 1501, 4, 1.8, plastic=0.05)
    for k, steps in enumerate((3, 1, 25, 2, 7, 19, 40, 1, 1, 30)):
        gb.set_schedule("step" if k % 2 else "persistent")
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps))
    gb.check()


@pytest.mark.parametrize("top", [32_767, 32_768])
def test_input_sums_at_the_edge_of_sixteen_bits(torch, top):
    """Neighbouring neurons whose inputs of one step sum to +-top (every presynaptic neuron fires at once): the
    16-bit accumulators hold 32,767, one more takes the 32-bit ones; partial resets and the step engine
    in between."""
    from flyzero_b200.brain import LIFParams
    from flyzero_b200.gpu import BatchBrain

    n, B, pre = 601, 3, 200
    w = np.zeros((n, n), np.float32)
    rng = np.random.default_rng(top)
    for k, col in enumerate((400, 401, 402, 403, 599, 600)):
        size = rng.multinomial(top - pre, np.full(pre, 1.0 / pre)) + 1
        w[:pre, col] = size * (1 if k % 3 else -1)
    w[:pre, 300:390] = rng.integers(-9, 9, (pre, 90))
    gb = BatchBrain(sp.csr_matrix(w), LIFParams(), batch=B, seed=4)
    eo = O.EngineOracle(sp.csr_matrix(w), O.Params(), batch=B, seed=4)
    gb.set_schedule("persistent")
    assert gb.info().epoch == (6 if top <= 32_767 else 4)
    idx = np.arange(pre)
    gb.set_input(idx, 20_000.0)                          # p > 1: every input neuron is kicked in every step
    j = eo.slots(idx)
    eo.p_ext[:, j] = np.float32(20_000.0) * np.float32(0.1 / 1000.0)
    for k, steps in enumerate((20, 7, 30, 25, 3, 40)):
        if k == 2:
            gb.set_schedule("step")
        if k == 3:
            gb.reset([1])
            eo.reset_flies([1])
            gb.set_schedule("persistent")
        if k == 4:
            gb.reset([0, 2])
            eo.reset_flies([0, 2])
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps))
    gb.check()


@pytest.mark.parametrize("integral", [True, False], ids=["counts", "float"])
@pytest.mark.parametrize("n,B,delay", [(127, 9, 1.8), (1003, 63, 1.8), (2001, 5, 0.5), (30_011, 6, 1.8)])
def test_stops_at_every_step_of_an_epoch(torch, n, B, delay, integral):
    """Instances that stop before, at and inside the epochs of a run, among others that do not: each takes its own
    number of steps of an epoch, and a stopped one stays as it was."""
    gb, eo = _pair(torch, n, B, delay, integral=integral, plastic=0.05, bias=0.03)
    _same(gb, eo, gb.run_steps(25), eo.run_steps(25))
    left = np.where(np.arange(B) % 5 == 4, -1, np.arange(B) % 29)
    gb.set_run_length(left)
    stop = np.where(left < 0, 2 ** 62, eo.t + left).astype(np.int64)
    for steps in (16, 1, 20):
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps, stop_tick=stop))
    ended = np.flatnonzero(left >= 0)
    gb.reset(ended)
    eo.reset_flies(list(ended))
    gb.set_run_length(np.full(B, -1))
    _same(gb, eo, gb.run_steps(31), eo.run_steps(31))
    gb.check()
