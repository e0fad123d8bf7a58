"""The persistent engine's pushes, two work items to a warp: rows whose lengths lie at the edges of a lane's
entries, of half a warp's and of an item, in odd and even numbers, bit for bit against the oracle."""

import numpy as np
import pytest
import scipy.sparse as sp

import oracle as O
from test_epochs_gpu import _same, torch  # noqa: F401

pytestmark = pytest.mark.gpu

LENGTHS = (0, 1, 7, 8, 9, 127, 128, 129, 136, 255, 256, 257, 384, 385, 513)


@pytest.mark.parametrize("integral", [True, False], ids=["counts", "float"])
@pytest.mark.parametrize("firing,hz", [(1, 20_000.0), (31, 20_000.0), (33, 20_000.0), (900, 400.0), (900, 20_000.0)])
def test_rows_of_every_length(torch, firing, hz, integral):  # noqa: F811
    from flyzero_b200.brain import LIFParams
    from flyzero_b200.gpu import BatchBrain

    n, B = 901, 3
    rng = np.random.default_rng(firing)
    rows, cols = [], []
    for i in range(n):
        k = LENGTHS[i % len(LENGTHS)]
        rows += [i] * k
        cols += list(rng.choice(n, k, replace=False))
    size = rng.integers(1, 5, len(rows)) if integral else rng.uniform(0.3, 4.0, len(rows))
    w = sp.csr_matrix(((size * rng.choice([1.0, -1.0], len(rows))).astype(np.float32), (rows, cols)), (n, n))
    gb = BatchBrain(w, LIFParams(), batch=B, seed=1)
    eo = O.EngineOracle(w, O.Params(), batch=B, seed=1)
    gb.set_schedule("persistent")
    idx = np.sort(rng.choice(n, firing, replace=False))
    gb.set_input(idx, hz)
    j = eo.slots(idx)
    eo.p_ext[:, j] = np.float32(hz) * np.float32(0.1 / 1000.0)
    for steps in (1, 40, 33):
        _same(gb, eo, gb.run_steps(steps), eo.run_steps(steps))
    gb.check()
