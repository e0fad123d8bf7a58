"""The schedules that autotune times are different ones: `lanes` is the step engine's, so the persistent engine
is listed once."""

from types import SimpleNamespace

import pytest

from flyzero_b200.gpu import BatchBrain


@pytest.mark.parametrize("group,f64,persistent", [(16, 0, 1), (0, 0, 0), (16, 1, 0)])
def test_each_schedule_is_listed_once(group, f64, persistent):
    cands = BatchBrain.schedule_candidates(SimpleNamespace(info=lambda: SimpleNamespace(group=group, f64=f64)))
    assert len(set(cands)) == len(cands)
    assert [c[0] for c in cands].count("persistent") == persistent
    assert [c for c in cands if c[0] == "step"] == [("step", "push", 8), ("step", "push", 32), ("step", "pull", 8)]
