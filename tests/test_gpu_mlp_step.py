"""The training step's kernels (csrc/rc_mlp.cu, needs a GB300): rc_mlp_train
draws its batches in layer 0 and ends a step with one launch that reduces the
gradient, applies Adam and packs the weights.  Against the same steps made of
rc_mlp_gradient and rc_mlp_adam on batches drawn here, for batches of one tile,
odd numbers of tiles and the most sample chunks.  After one step only the bias
corrections differ (powf on the device, 1 ulp of 1 - beta^k: 6e-7 of the
update, at most lr); the losses of four steps differ by the BF16 roundings of
weights that this moves."""
import math

import numpy as np
import pytest

from test_gpu_mlp import MEAN, STD, raw_samples

pytestmark = pytest.mark.gpu


def drawn(seed, it, batch, n):
    m = (1 << 64) - 1
    z = [(seed + 0x9E3779B97F4A7C15 * (it * batch + i + 1)) & m for i in range(batch)]
    z = [((v ^ (v >> 30)) * 0xBF58476D1CE4E5B9) & m for v in z]
    z = [((v ^ (v >> 27)) * 0x94D049BB133111EB) & m for v in z]
    return np.array([(v ^ (v >> 31)) % n for v in z])


@pytest.mark.parametrize("batch", [128, 384, 8320, 16384])
def test_step_equals_gradient_and_adam(batch):
    import torch
    from rocketcombustor_gb300 import surrogate
    n, lr, lr_end, seed = 20000, 3e-3, 3e-4, 7
    x = torch.tensor(raw_samples(n, batch), device="cuda")
    t = torch.rand(n, 4, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    for steps in (1, 4):
        a, b = surrogate.MLP(seed=5), surrogate.MLP(seed=5)
        for m in (a, b):
            m.set_norm(MEAN, STD)
        hist = a.train(x, t, steps=steps, batch=batch, lr=lr, lr_end=lr_end, seed=seed, log_every=1)
        losses = []
        for k in range(steps):
            j = torch.tensor(drawn(seed, k, batch, n), device="cuda")
            g, loss = b.gradient(x[j].contiguous(), t[j].contiguous())
            losses.append(float(loss))
            b.adam(g, lr_end + 0.5 * (lr - lr_end) * (1 + math.cos(math.pi * k / max(steps - 1, 1))))
        assert np.allclose([h[1] for h in hist], losses, rtol=1e-6 if steps == 1 else 1e-3, atol=0)
        if steps == 1:
            p, q = a.get_params(), b.get_params()
            assert np.abs(p - q).max() <= 1e-6 * lr + 2 * np.spacing(np.abs(q).max())
        a.close()
        b.close()
