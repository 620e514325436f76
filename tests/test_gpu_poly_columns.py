"""The cp polynomial columns that the kernels evaluate (needs a GB300).

Columns of zeros are left out of the sums (csrc/rc_thermo.cuh); the oracle
adds all seven.  The states are equal bit for bit whichever columns hold
coefficients: the constant alone, the first or the last column first, a gap,
all seven, and different ones below and above the critical temperature.
"""
import numpy as np
import pytest

import oracle
import rocketcombustor_gb300 as rc
from rocketcombustor_gb300 import cases

pytestmark = pytest.mark.gpu

# a1/T^2, a2/T, a3, a4 T, a5 T^2, a6 T^3, a7 T^4: each a few percent of cp/R or less at 1000-3500 K
SIZE = np.array([2.0e3, 5.0, 3.6, 3.0e-5, 5.0e-9, 1.0e-12, 2.0e-16])


@pytest.mark.parametrize("low,high", [((2,), (2,)), ((0, 2), (0, 2)), ((1, 2), (1, 2)), ((2, 4, 6), (2, 4, 6)),
                                      ((0, 1, 2, 3, 4, 5, 6), (0, 1, 2, 3, 4, 5, 6)), ((2, 3), (2, 5, 6))])
def test_columns_bit_identical(tmp_path, low, high):
    d = str(tmp_path)
    cases.make_case(d, "t2")
    rng = np.random.default_rng(31)
    tab = [np.zeros((4, 7)), np.zeros((4, 7))]
    for t, cols in zip(tab, (low, high)):
        for j in cols:
            t[:, j] = SIZE[j] * rng.uniform(0.9, 1.1, 4)
    # the critical temperature in the middle of the field, so that both ranges are met
    cases.write_thermo(d, tab[0], tab[1], [0.0, 0.0, -29084.98253056227, 0.0], trange=(200.0, 3000.0, 60000.0))
    o, s = oracle.Oracle(d, threads=4), rc.Solver(rc.Case(d))
    o.run(4)
    s.run(4)
    PA, WA = s.get_state()
    assert np.array_equal(PA, o.array("PA")) and np.array_equal(WA, o.array("WA"))
