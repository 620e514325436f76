"""rc_chem_integrate in a stream capture (needs a GB300): a captured call, larger
than the calls before it, neither synchronises nor allocates, and its replay
after larger calls still has its own work space.  Growing calls on one context
are those of fresh contexts."""
import numpy as np
import pytest

import oracle
import rocketcombustor_gb300 as rc
from conftest import make_case
from test_chem import states

pytestmark = pytest.mark.gpu


def inputs(case_root, n, seed):
    import torch
    pool = states(oracle.Oracle(make_case(case_root, "t2"), threads=4), 2048, 9)
    rng = np.random.default_rng(seed)
    P = torch.tensor(pool[rng.integers(0, len(pool), n)].T.copy(), dtype=torch.float64, device="cuda")
    return P, torch.tensor(10 ** rng.uniform(-10, -6, n), device="cuda")


def call(s, P, dt, out, nsub):
    return rc.load().rc_chem_integrate(s._h, P.data_ptr(), dt.data_ptr(), P.shape[1], out.data_ptr(), nsub.data_ptr(),
                                       0.05, 200)


@pytest.mark.parametrize("warm", [32, 30000])
def test_replay_after_larger_calls(case_root, warm):
    import torch
    c = rc.Case(make_case(case_root, "t2"))
    n = 40000 if warm == 32 else warm  # larger than any call before it, or as large
    P, dt = inputs(case_root, n, 1)
    ref, nref = rc.Solver(c).chem_integrate(P, dt)
    st = torch.cuda.Stream()
    s = rc.Solver(c, stream=st.cuda_stream)
    s.chem_integrate(P[:, :warm], dt[:warm])
    out, nsub = torch.zeros_like(P), torch.zeros(n, dtype=torch.int32, device="cuda")
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=st):
        assert call(s, P, dt, out, nsub) == 0
    for larger in (n + 1, 4 * n):
        s.chem_integrate(*inputs(case_root, larger, larger))
        # what a freed list would be given to
        guard = [torch.full((k << 20,), 7, dtype=torch.uint8, device="cuda") for k in (1, 2, 4, 8, 16, 32)]
        out.zero_()
        nsub.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            g.replay()
        s.sync()
        assert torch.equal(out, ref) and torch.equal(nsub, nref)
        assert all(bool((x == 7).all()) for x in guard)
        del guard
    s.close()


def test_growing_calls(case_root):
    import torch
    c = rc.Case(make_case(case_root, "t2"))
    s = rc.Solver(c)
    for n in (100, 20000, 20001, 50000, 30000, 200000):
        P, dt = inputs(case_root, n, n)
        fresh = rc.Solver(c)
        a, b = s.chem_integrate(P, dt), fresh.chem_integrate(P, dt)
        assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
        fresh.close()
    s.close()
