"""The schedule that rc_init chooses by itself, on both sides of its rules'
lines (the smallest mesh, a mesh of few levels, levels that fill one compact
group of an SM and two, levels that fill the GPU) and of the block count's,
against the per-level sweeps: the same states bit for bit."""
import numpy as np
import pytest

import rocketcombustor_gb300 as rc
from conftest import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [rc.RC_PREC_FP64, rc.RC_PREC_MIXED])
@pytest.mark.parametrize("name,over", [("c1", {"nx": 4, "ny": 2}), ("t2", {}),
                                       ("c2", {"nx": 60, "ny": 10, "order": "random"}),
                                       ("c1", {"nx": 9000, "ny": 4}), ("c2", {"nx": 3000, "ny": 4}),
                                       ("c2", {"nx": 200, "ny": 150, "order": "colored"})])
def test_chosen_schedule_equals_per_level_sweeps(case_root, precision, name, over, monkeypatch):
    c = rc.Case(make_case(case_root, name, **over))
    states = []
    for sched in (None, "levels"):
        if sched:
            monkeypatch.setenv("RC_LUSGS_SCHEDULE", sched)
        else:
            monkeypatch.delenv("RC_LUSGS_SCHEDULE", raising=False)
        s = rc.Solver(c, precision=precision)
        s.run(12)
        states.append(s.get_state())
        s.close()
    assert np.array_equal(states[0][0], states[1][0])
    assert np.array_equal(states[0][1], states[1][1])
