"""The integrator's lists when they are too short (needs a GB300): more states
that need more attempts than the first round gives them than a list has places
(2^20), so that some stay in their lanes.  Each state's result and substep count
are those of a call in one round."""
import numpy as np
import pytest

import oracle
import rocketcombustor_gb300 as rc
from conftest import make_case
from test_chem import states

pytestmark = pytest.mark.gpu

PLACES, FIRST_ROUND = 1 << 20, 16


def test_more_long_states_than_places(case_root):
    import torch
    d = make_case(case_root, "t2")
    s = rc.Solver(rc.Case(d))
    # one round: at most 128 states per SM
    P = torch.tensor(states(oracle.Oracle(d, threads=4), 16384, 9).T.copy(), dtype=torch.float64, device="cuda")
    dt = torch.tensor(10 ** np.random.default_rng(5).uniform(-7, -5, P.shape[1]), device="cuda")
    out, nsub = s.chem_integrate(P, dt, 0.005, 2000)
    # accepted substeps only: each of these takes more attempts than that
    long = torch.nonzero(nsub > FIRST_ROUND)[:, 0]
    assert long.numel() > 1000
    n = PLACES + 150_000
    j = long[torch.randint(long.numel(), (n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(2))]
    o1, n1 = s.chem_integrate(P[:, j].contiguous(), dt[j].contiguous(), 0.005, 2000)
    assert torch.equal(n1, nsub[j])
    assert torch.equal(o1, out[:, j])
