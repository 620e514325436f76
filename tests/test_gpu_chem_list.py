"""The integrator in the steady iteration on more cells than one block per SM
holds (needs a GB300): the integrated source's rounds over sorted cells, and
those over the surrogate's list of cells that it hands back.  With an error
indicator that rejects every cell the list holds them all, and the source is
the integrated one.  A list costs at most two launches more than one round,
since it is usually empty."""
import numpy as np
import pytest

import oracle
import rocketcombustor_gb300 as rc
from conftest import make_case
from test_gpu_mlp import MEAN, STD

pytestmark = pytest.mark.gpu


def surrogate_solver(c, tol):
    from rocketcombustor_gb300 import surrogate
    net = surrogate.MLP(seed=7)
    net.set_norm(MEAN, STD)
    s = rc.Solver(c)
    s.set_surrogate(net, tol)
    s.set_chemistry(rc.RC_CHEM_SURROGATE, 0.005, 2000)
    return s


def test_integrated_source_in_rounds_bit_identical_to_oracle(case_root):
    d = make_case(case_root, "c2", nx=300, ny=50)
    s = rc.Solver(rc.Case(d))
    s.set_chemistry(rc.RC_CHEM_INTEGRATED)
    s.run(2)
    o = oracle.Oracle(d, threads=oracle.Oracle.max_threads())
    o.set_chemistry(1)
    o.run(2)
    PA, WA = s.get_state()
    assert np.array_equal(s.chem_substeps(), o.chem_nsub())
    assert np.array_equal(PA, o.array("PA")) and np.array_equal(WA, o.array("WA"))


# 1.5 and 6 blocks of cells per SM: fewer and more items than the launch has lanes
@pytest.mark.parametrize("nx,ny", [(300, 50), (600, 100)])
def test_listed_cells_equal_the_integrated_source(case_root, nx, ny):
    c = rc.Case(make_case(case_root, "c2", nx=nx, ny=ny))
    ref = rc.Solver(c)
    ref.set_chemistry(rc.RC_CHEM_INTEGRATED, 0.005, 2000)
    s = surrogate_solver(c, 1e-12)
    for x in (ref, s):
        x.run(3)
    assert s.surrogate_stats() == (0, c.NE)
    assert np.array_equal(s.chem_substeps(), ref.chem_substeps())
    a, b = s.get_state(), ref.get_state()
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_launches_of_an_iteration(case_root):
    def launches(nx, ny):
        s = surrogate_solver(rc.Case(make_case(case_root, "c2", nx=nx, ny=ny)), 0.02)
        s.lu_sgs_stage(1)
        before = s.stats()["kernel_launches"]
        s.lu_sgs_stage(2)
        n = s.stats()["kernel_launches"] - before
        s.close()
        return n

    assert launches(300, 50) <= launches(60, 10) + 2
