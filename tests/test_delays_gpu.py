"""The persistent engine at every synaptic delay from 3 steps, bit for bit against the oracle: epochs of each
length, listed late or at their own end, with accumulators of each width; plastic and biased neurons,
instances that stop, more spikes than a CTA's buffer holds, and both engines in turn."""

import numpy as np
import pytest

from test_epochs_gpu import _pair, _same, torch  # noqa: F401

pytestmark = pytest.mark.gpu

# n_delay -> steps between barriers with 16-bit accumulators (at most 4 with wider ones)
EPOCH = {3: 1, 4: 2, 5: 2, 6: 3, 7: 3, 8: 4, 9: 4, 10: 5, 11: 5, 12: 6, 13: 6, 14: 6, 15: 5, 16: 5, 17: 5, 18: 6, 40: 6}


@pytest.mark.parametrize("integral", [True, False], ids=["counts", "float"])
@pytest.mark.parametrize("n_delay", sorted(EPOCH))
def test_every_delay_matches_the_oracle(torch, n_delay, integral):  # noqa: F811
    gb, eo = _pair(torch, 1003, 7, n_delay * 0.1, integral=integral, plastic=0.05, bias=0.03)
    assert gb.n_delay == n_delay
    for steps in (1, 2, 53, 7, 40):
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps))
    if integral:
        assert gb.info().epoch == EPOCH[n_delay]
    left = np.array([0, 1, 3, 7, 12, 25, -1])
    gb.set_run_length(left)
    stop = np.where(left < 0, 2 ** 62, eo.t + left).astype(np.int64)
    _same(gb, eo, gb.run_steps(33), eo.run_steps(33, stop_tick=stop))
    gb.check()


@pytest.mark.parametrize("n_delay", [3, 4, 5, 8, 9, 10])
def test_wide_accumulators_at_short_delays(torch, n_delay):  # noqa: F811
    """Counts whose sums leave 16 bits (32-bit accumulators), recorded step by step."""
    import scipy.sparse as sp

    import oracle as O
    from flyzero_b200.brain import LIFParams
    from flyzero_b200.gpu import BatchBrain

    n, B = 401, 5
    rng = np.random.default_rng(n_delay)
    w = np.zeros((n, n), np.float32)
    w[:150, 200:] = rng.integers(-3, 9, (150, n - 200))
    w[:150, 399] = 300                                   # 45,000 if all fire at once
    gb = BatchBrain(sp.csr_matrix(w), LIFParams(delay=n_delay * 0.1), batch=B, seed=2)
    eo = O.EngineOracle(sp.csr_matrix(w), O.Params(delay=n_delay * 0.1), batch=B, seed=2)
    gb.set_schedule("persistent")
    gb.set_input(np.arange(150), 3000.0)
    j = eo.slots(np.arange(150))
    eo.p_ext[:, j] = np.float32(3000.0) * np.float32(0.1 / 1000.0)
    for steps in (1, 30, 5, 22):
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps))
    gb.check()


@pytest.mark.parametrize("n_delay", [4, 5, 8, 12])
def test_full_buffers_where_epochs_list_their_own_spikes(torch, n_delay):  # noqa: F811
    gb, eo = _pair(torch, 40_000, 8, n_delay * 0.1, degree=3, driven=1.0, hz=20_000.0)
    assert 8 * 40_000 / gb.info().ctas > 2048
    for steps in (9, 30):
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps))
    gb.check()


@pytest.mark.parametrize("n_delay", [3, 4, 5, 10, 16])
def test_engines_in_turn_at_short_delays(torch, n_delay):  # noqa: F811
    gb, eo = _pair(torch, 1501, 4, n_delay * 0.1, plastic=0.05)
    for k, steps in enumerate((3, 1, 25, 2, 7, 19, 40, 1, 1, 30)):
        gb.set_schedule("step" if k % 2 else "persistent")
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps))
    gb.check()


@pytest.mark.parametrize("n_delay", [5, 18])
def test_more_inputs_than_shared_memory_has_room_for(torch, n_delay):  # noqa: F811
    """Nearly as many pairs as the chip holds, all of them inputs: most thresholds stay in global memory."""
    gb, eo = _pair(torch, 39_990, 62, n_delay * 0.1, degree=2, driven=1.0, hz=300.0)
    info = gb.info()
    assert info.group == 62 and 62 * 39_990 / info.ctas > 16_000
    for steps in (7, 9):
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps))
    gb.check()


@pytest.mark.parametrize("n_delay", [3, 5, 18])
def test_stops_on_one_engine_then_the_other(torch, n_delay):  # noqa: F811
    """Instances that stop (one with input still on its way) while one engine runs, then the other takes over: what
    is in flight follows, what a stopped instance left behind does not come back after its reset."""
    gb, eo = _pair(torch, 1201, 6, n_delay * 0.1, plastic=0.05, bias=0.03)

    def run(engine, steps, stop=None):
        gb.set_schedule(engine)
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps) if stop is None else eo.run_steps(steps, stop_tick=stop))

    for first, second in (("step", "persistent"), ("persistent", "step"), ("step", "persistent")):
        run(first, 25)
        left = np.array([0, 1, 4, 9, 17, -1])                      # instance 0 stops with the next tick's input pushed
        gb.set_run_length(left)
        stop = np.where(left < 0, 2 ** 62, eo.t + left).astype(np.int64)
        run(first, 11, stop)
        run(second, 13, stop)
        run(first, 2, stop)
        ended = [0, 1, 2, 3, 4]
        gb.reset(ended)
        eo.reset_flies(ended)
        gb.set_run_length(np.full(6, -1))
        run(second, 27)
    gb.check()


def test_device_memory_of_a_count_network(torch):  # noqa: F811
    """The delay line's bytes for 16-bit sums: 12 slots of 2 and 2 of 4 per pair, n_delay + 1 lists of every pair."""
    from flyzero_b200.brain import LIFParams
    from flyzero_b200.gpu import BatchBrain
    from test_epochs_gpu import _net

    n, B = 20_000, 8
    w = _net(n, 8, 1, True)
    a, b = (BatchBrain(w, LIFParams(), batch=B * k).info() for k in (1, 2))
    pair = 9 + 4 + 12 * 2 + 2 * 4 + 19 * 8             # state, ext_idx aside; a row is one item
    assert b.epoch == 6 and b.bytes_device - a.bytes_device <= 1.02 * B * n * pair
