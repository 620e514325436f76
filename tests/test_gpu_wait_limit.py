"""The bound on the waits inside the sweeps' launches (rc_set_wait_limit, units
of 256 ns; needs a GB300), in the compact dataflow launches that rc_init
chooses on most meshes.  A limit that covers the launch is enough, although
some warps wait through a whole sweep on polls that take a tenth of a unit;
a limit of 1 ends every wait, with RC_ERR_SYNC, and leaves the context usable."""
import numpy as np
import pytest

import oracle
import rocketcombustor_gb300 as rc
from conftest import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sched", ["flowc", "flowc2"])
@pytest.mark.parametrize("precision", [rc.RC_PREC_FP64, rc.RC_PREC_MIXED])
def test_limit_that_covers_the_launch_is_enough(case_root, precision, sched, monkeypatch):
    import torch
    monkeypatch.setenv("RC_LUSGS_SCHEDULE", sched)
    s = rc.Solver(rc.Case(make_case(case_root, "c2", nx=300, ny=50)), precision=precision)
    s.run(3)
    s.sync()
    stream = torch.cuda.ExternalStream(s.stream())
    a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    a.record(stream)
    for it in range(10):
        s.lu_sgs_stage(it + 4)
    b.record(stream)
    s.sync()
    # one iteration, of which the sweeps' launch is a part
    s.set_wait_limit(int(a.elapsed_time(b) / 10 * 1e-3 / 256e-9) + 1)
    s.run(10)
    s.sync()
    s.close()


@pytest.mark.parametrize("precision", [rc.RC_PREC_FP64, rc.RC_PREC_MIXED])
def test_flowc_wait_timeout_is_reported(case_root, precision, monkeypatch):
    monkeypatch.setenv("RC_LUSGS_SCHEDULE", "flowc")
    d = make_case(case_root, "t2")
    c = rc.Case(d)
    s = rc.Solver(c, precision=precision)
    s.set_wait_limit(1)
    s.lu_sgs_stage(1)
    with pytest.raises(rc.RcError) as e:
        s.sync()
    assert e.value.code & 64
    s.clear_error()
    s.set_wait_limit(1 << 24)
    s.set_state(c.array("PA"), c.array("WA"))
    s.run(5)
    PA, WA = s.get_state()
    if precision == rc.RC_PREC_FP64:
        o = oracle.Oracle(d, threads=4)
        o.run(5)
        P0, W0 = o.array("PA"), o.array("WA")
    else:
        clean = rc.Solver(c, precision=precision)
        clean.set_state(c.array("PA"), c.array("WA"))
        clean.run(5)
        P0, W0 = clean.get_state()
        clean.close()
    assert np.array_equal(PA, P0) and np.array_equal(WA, W0)
    s.close()
