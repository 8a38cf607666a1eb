"""First calls on new contexts while several processes share the GPU: what the setup
copied to the device (descriptors, tables, tensor maps, features) has arrived
before the first kernel reads it, however late the copies run."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import sys
import numpy as np
from fgpu import PERIODIC, RBF, SUM, Engine, loglik_batch
from fgpu.gpr import set_trailing_update
set_trailing_update(sys.argv[1])
seen = set()
for k in range(12):
    n = 1000 + 64 * (k % 3)
    rng = np.random.default_rng(n)
    X = rng.normal(2.0, 0.3, size=(n, 8))
    X[:, 7] = rng.uniform(-np.pi, np.pi, size=n)
    e = Engine(X, np.cos(X[:, 0]), np.zeros(n), [RBF, 7, 1, 2, 3, 4, 5, 6, 7, PERIODIC, 1, 8, SUM], 0, 1e-3, False)
    th = np.full(8, 0.4)
    first = e.grad(th) if k % 2 else e.loglik(th)
    ll, info = e.loglik(th)
    lb, ib = loglik_batch([e] * 3, [th] * 3)
    assert first[0] == ll and first[-1] == info == 0, (k, first, ll, info)
    assert np.all(ib == 0) and np.all(lb == lb[0]) and abs(lb[0] - ll) <= 1e-12 * abs(ll), (k, lb, ib, ll)
    seen.add((n, ll))
    e.close()
assert len(seen) == 3, seen
"""


@pytest.mark.parametrize("mode", ["fp64", "tcgen05"])
def test_first_calls_of_several_processes(mode, lib):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=os.path.join(root, "ferebus-v7_gb300"))
    ps = [subprocess.Popen([sys.executable, "-c", CHILD, mode], env=env, stderr=subprocess.PIPE, text=True)
          for _ in range(5)]
    err = [p.communicate(timeout=300)[1] for p in ps]
    assert all(p.returncode == 0 for p in ps), "\n".join(err)
