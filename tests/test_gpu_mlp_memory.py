"""A gradient call that there is no memory for (needs a GB300): it returns an
error and leaves the network usable, with work buffers of its own in the next
call."""
import pytest

import rocketcombustor_gb300 as rc
from test_gpu_mlp import MEAN, STD, raw_samples

pytestmark = pytest.mark.gpu


def test_gradient_after_a_batch_too_large():
    import torch
    from rocketcombustor_gb300 import surrogate
    m = surrogate.MLP(seed=3)
    m.set_norm(MEAN, STD)
    xs = torch.tensor(raw_samples(4096, 1), device="cuda")
    ts = torch.rand(4096, 4, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    x, t = xs[:1024].contiguous(), ts[:1024].contiguous()
    g0, l0 = m.gradient(x, t)
    d = torch.empty_like(g0)
    # over a terabyte of pre-activations; the call ends before it reads a sample
    n = (1 << 31) - 128
    st = rc.load().rc_mlp_gradient(m.handle, x.data_ptr(), t.data_ptr(), n, d.data_ptr(), None, None)
    assert st != 0
    g1, l1 = m.gradient(x[:512].contiguous(), t[:512].contiguous())
    g2, l2 = m.gradient(x, t)
    assert torch.equal(g0, g2) and float(l0) == float(l2)
    assert bool(torch.isfinite(g1).all())
    # and after a larger one
    hist = m.train(xs, ts, steps=2, batch=2048, log_every=1)
    assert all(v == v for _, v in hist)
    m.close()
