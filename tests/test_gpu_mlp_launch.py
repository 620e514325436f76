"""A training call of which a later step cannot be launched (needs a GB300; the
failure comes from a stand-in for cudaGraphLaunch): it returns the error, and
the network infers with the parameters that the steps before it left."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

RUN = """
import torch
import rocketcombustor_gb300 as rc
from rocketcombustor_gb300 import surrogate
from test_gpu_mlp import MEAN, STD, raw_samples

x = torch.tensor(raw_samples(4096, 1), device="cuda")
t = torch.rand(4096, 4, device="cuda")
m = surrogate.MLP(seed=3)
m.set_norm(MEAN, STD)
p = m.get_params()
try:
    m.train(x, t, steps=5, batch=1024, lr=1e-2)
    raise SystemExit("no error")
except rc.RcError:
    pass
q = m.get_params()
assert abs(p - q).max() > 1e-3  # two steps
f = surrogate.MLP(seed=4)
f.set_norm(MEAN, STD)
f.set_params(q)
assert torch.equal(m.forward(x), f.forward(x))
m.train(x, t, steps=2, batch=1024)
f.set_params(m.get_params())
assert torch.equal(m.forward(x), f.forward(x))
print("as the parameters")
"""


def test_inference_follows_the_steps_that_ran(tmp_path):
    lib = str(tmp_path / "fail_launch.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", lib, os.path.join(HERE, "cuda", "fail_graph_launch.c"), "-ldl"],
                   check=True)
    env = dict(os.environ, LD_PRELOAD=lib, RC_FAIL_LAUNCH="3",
               PYTHONPATH=os.pathsep.join([os.path.dirname(HERE), HERE, os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", RUN], capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0 and "as the parameters" in r.stdout, r.stdout + r.stderr
