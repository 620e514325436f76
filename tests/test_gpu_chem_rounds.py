"""The integrator's rounds (csrc/rc_chem.cu, needs a GB300): calls with more
states than one block per SM holds park their long states and take them up
again in later launches.  Counts around that line, above the launch's lanes
(a round then ends with its queue), and above the lists' million places: each
state's result and substep count are those of calls that run in one round."""
import numpy as np
import pytest

import oracle
import rocketcombustor_gb300 as rc
from conftest import make_case
from test_chem import states

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_sm", [128, 129, 400, 1000, 7700])
def test_rounds_equal_one_round(case_root, per_sm):
    import torch
    d = make_case(case_root, "t2")
    s = rc.Solver(rc.Case(d))
    nsm = torch.cuda.get_device_properties(0).multi_processor_count
    n, part = nsm * per_sm, nsm * 128
    rng = np.random.default_rng(per_sm)
    P = states(oracle.Oracle(d, threads=4), 4096, 9)
    P = torch.tensor(P[rng.integers(0, len(P), n)].T.copy(), dtype=torch.float64, device="cuda")
    dt = 10 ** rng.uniform(-10, -6 if per_sm < 2000 else -8, n)
    dt[rng.random(n) < 0.1] = 0.0
    dt = torch.tensor(dt, device="cuda")
    out, nsub = s.chem_integrate(P, dt)
    for a in range(0, n, part):
        o1, n1 = s.chem_integrate(P[:, a:a + part].contiguous(), dt[a:a + part].contiguous())
        assert torch.equal(nsub[a:a + part], n1)
        assert torch.equal(out[:, a:a + part], o1)
