"""A solver on the caller's streams (rc_set_stream; needs a GB300): the time step
and the diagonal run on a stream of the context beside them, the integrated
source on another, joined in the captured stage and in the BDF2 inner iteration.
The states are those of a solver on its own stream, also when the caller's
stream changes between stages and when the caller's stream has other work."""
import numpy as np
import pytest

import rocketcombustor_gb300 as rc
from conftest import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,chem", [(rc.RC_PREC_FP64, rc.RC_CHEM_EXPLICIT), (rc.RC_PREC_MIXED, rc.RC_CHEM_EXPLICIT),
                                            (rc.RC_PREC_FP64, rc.RC_CHEM_INTEGRATED)])
def test_stage_on_the_callers_streams(case_root, precision, chem):
    import torch
    c = rc.Case(make_case(case_root, "c2", nx=60, ny=10))
    ref = rc.Solver(c, precision=precision)
    ref.set_chemistry(chem)
    ref.run(9)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    s = rc.Solver(c, precision=precision, stream=a.cuda_stream)
    s.set_chemistry(chem)
    busy = torch.zeros(1 << 24, device="cuda")
    for k, st in enumerate((a, b, a)):
        s.sync()
        assert rc.load().rc_set_stream(s._h, st.cuda_stream) == 0
        with torch.cuda.stream(st):
            for _ in range(20):
                busy += 1.0
        for it in range(3):
            s.lu_sgs_stage(3 * k + it + 1)
    PA, WA = s.get_state()
    P0, W0 = ref.get_state()
    assert np.array_equal(PA, P0) and np.array_equal(WA, W0)
    s.close()


def test_bdf2_on_the_callers_stream(case_root):
    import torch
    c = rc.Case(make_case(case_root, "c2u", nx=40, ny=8))
    u = c.unsteady
    ref, st = rc.Solver(c), torch.cuda.Stream()
    s = rc.Solver(c, stream=st.cuda_stream)
    for k in (1, 2):
        n = [x.bdf2_stage(k, u["dt"], u["inner_loop"], u["rel_tol"]) for x in (ref, s)]
        assert n[0] == n[1]
    a, b = s.get_state(), ref.get_state()
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    s.close()
