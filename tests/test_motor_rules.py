"""BatchMotor.update asks the button rule that is in force: the class's own (over columns), a subclass's, or one set
on the instance (slot by slot)."""

from types import SimpleNamespace

import numpy as np
import pytest

from flyzero_b200 import motor
from flyzero_b200.motor import BatchMotor, MotorParams, READOUT


class Half(BatchMotor):
    def buttons(self, r, k):
        return {"slot": k, "first": float(r[0])}


@pytest.mark.parametrize("kind", ["own", "subclass", "instance"])
def test_update_asks_the_rule_in_force(monkeypatch, kind):
    torch = pytest.importorskip("torch")
    rates = np.random.default_rng(1).uniform(0, 30, (7, len(READOUT))).astype(np.float32)
    m = object.__new__(Half if kind == "subclass" else BatchMotor)
    m.p, m.B, m.g, m.w, m.acc = MotorParams(), 7, SimpleNamespace(idx=None, ptr=None, n_groups=9), None, np.zeros((7, 2))
    m.rates_dev = torch.as_tensor(rates)
    m.brain = SimpleNamespace(_L=SimpleNamespace(fb_group_rates=lambda *a: 0), _h=None, device=None)
    monkeypatch.setattr(motor, "_stream", lambda dev: None)
    if kind == "instance":
        m.buttons = lambda r, k: {"slot": k, "first": float(r[0])}
    got = m.update(None, 16.6)
    want = [m.buttons(r, k) for k, r in enumerate(rates)]
    assert got == want and len(got) == 7
    if kind != "own":
        assert got[3] == {"slot": 3, "first": float(rates[3, 0])}
