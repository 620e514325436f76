"""The integrator's work queue (csrc/rc_chem.cu, needs a GB300): lanes take new
items as they finish old ones, so which warp integrates a state, and beside
which others, depends on the count.  Each state's result and substep count
equal the oracle's bit for bit: counts around a warp and a refill, states of
very uneven cost next to one another, and states with nothing to integrate."""
import numpy as np
import pytest

import oracle
import rocketcombustor_gb300 as rc
from conftest import make_case
from test_chem import states

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 31, 32, 33, 100, 700])
def test_queue_bit_identical(case_root, n):
    import torch
    d = make_case(case_root, "t2")
    o = oracle.Oracle(d, threads=4)
    s = rc.Solver(rc.Case(d))
    P = states(o, n, 40 + n)
    rng = np.random.default_rng(n)
    dt = 10 ** rng.uniform(-10, -5, n)
    dt[rng.random(n) < 0.1] = 0.0
    ref, nref = o.chem_integrate(P, dt)
    out, nsub = s.chem_integrate(torch.tensor(P.T.copy(), dtype=torch.float64, device="cuda"),
                                 torch.tensor(dt, device="cuda"))
    assert np.array_equal(nsub.cpu().numpy(), nref)
    assert np.array_equal(out.cpu().numpy().T, ref)
