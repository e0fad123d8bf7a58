"""The step engine's launches, bit for bit against the oracle: a delay of one step (the spikes of a step are pushed by a
second launch), of two and more (one launch pushes and advances), rows that end inside a block,
both state types, every width of a work item's lane group, plastic synapses, instances that stop, and pull
propagation in between."""
import numpy as np
import pytest
import scipy.sparse as sp

import oracle as O

pytestmark = pytest.mark.gpu


def _pair(n, B, delay, real, integral, seed=5):
    from flyzero_b200.brain import LIFParams
    from flyzero_b200.gpu import BatchBrain

    rng = np.random.default_rng(seed)
    degree = min(n, 12)
    w = sp.coo_matrix((np.ones(n * degree), (np.repeat(np.arange(n), degree), rng.integers(0, n, n * degree))), (n, n)).tocsr()
    w.sum_duplicates()
    size = rng.integers(1, 9, w.nnz) if integral else rng.uniform(0.3, 9.0, w.nnz)
    w.data = (size * rng.choice([1.0, 1.0, -1.0], w.nnz)).astype(np.float32)
    pos = np.sort(rng.choice(w.nnz, max(1, w.nnz // 20), replace=False))
    gb = BatchBrain(w, LIFParams(delay=delay), batch=B, seed=seed, plastic_pos=pos, fp64=real is np.float64)
    eo = O.EngineOracle(w, O.Params(delay=delay), batch=B, plastic_pos=pos, seed=seed, real=real)
    idx = np.sort(rng.choice(n, max(1, n // 3), replace=False))
    rates = rng.uniform(0.0, 300.0, (B, len(idx))).astype(np.float32)
    gb.set_input(idx, rates)
    j = eo.slots(idx)
    eo.p_ext[:, j] = rates * np.float32(0.1 / 1000.0)
    return gb, eo


def _same(gb, eo, c, want):
    np.testing.assert_array_equal(c.cpu().numpy(), want)
    for name in ("v", "g", "ref"):
        np.testing.assert_array_equal(getattr(gb, name).cpu().numpy(), getattr(eo, name))


@pytest.mark.parametrize("real", [np.float32, np.float64])
@pytest.mark.parametrize("integral", [True, False], ids=["counts", "float"])
@pytest.mark.parametrize("n,B,delay", [(1, 1, 0.1), (255, 3, 0.1), (257, 5, 0.2), (1000, 7, 0.3), (4099, 17, 1.8)])
def test_step_launches_match_the_oracle(n, B, delay, integral, real):
    gb, eo = _pair(n, B, delay, real, integral)
    assert gb.n_delay == round(delay / 0.1)
    for k, (steps, lanes) in enumerate(((1, 8), (2, 16), (41, 32), (30, 8))):
        gb.set_schedule("step", lanes=lanes)
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps))
    left = np.where(np.arange(B) % 2, 5, -1)
    gb.set_run_length(left)
    stop = np.where(left < 0, 2 ** 62, eo.t + left).astype(np.int64)
    _same(gb, eo, gb.run_steps(23), eo.run_steps(23, stop_tick=stop))
    gb.check()


def test_several_tiles_per_block():
    gb, eo = _pair(20_011, 61, 1.8, np.float32, True)          # 79 x 61 tiles: two for each block, the last one ragged
    gb.set_schedule("step", lanes=8)
    _same(gb, eo, gb.run_steps(40), eo.run_steps(40))
    gb.check()


@pytest.mark.parametrize("delay", [0.1, 0.2, 1.8])
def test_pull_between_pushes(delay):
    gb, eo = _pair(777, 4, delay, np.float64, True)
    for prop, steps in (("push", 25), ("pull", 44), ("push", 30)):
        gb.set_schedule("step", prop)
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps))
    gb.check()
