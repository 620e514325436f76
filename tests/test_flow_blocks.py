"""The compact dataflow plan on few blocks (host only): every check of
rc_flow_plan_stats, the places of the neighbours among the block's last passes
among them, from one block that holds the whole mesh up to more blocks than
cells of a level."""
import numpy as np
import pytest

import rocketcombustor_gb300 as rc
from conftest import make_case


@pytest.mark.parametrize("nblocks", [1, 2, 7, 40, 300])
@pytest.mark.parametrize("name,over", [("t1", {}), ("s2t", {}), ("c2", {"nx": 60, "ny": 10, "order": "random"})])
def test_compact_plan_on_any_number_of_blocks(case_root, name, over, nblocks):
    c = rc.Case(make_case(case_root, name, **over))
    nei = c.array("Neighbor")
    face = c.array("NeighF")
    co = np.full((c.NE, 4), -1, np.int32)
    for q in range(4):
        f = face[:, q] - 1
        ok = f >= 0
        a, b = nei[f[ok], 0], nei[f[ok], 1]
        me = np.nonzero(ok)[0] + 1
        other = np.where(a == me, b, a)
        co[ok, q] = np.where(other > 0, other - 1, -1)
    for groups in (1, 2):
        st = rc.flow_plan_check(c.array("KFace"), co, nblocks, groups=groups, compact=True, nvar=c.NVar)
        assert st["passes_fwd"] >= st["levels_fwd"] and st["steps"] >= st["levels_fwd"]
