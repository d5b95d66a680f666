"""A root solve that ends in the reference's bisection, which can run its 10^6
iterations (EnergyMomentumTensor.cpp:48-111), runs it once: the fused stage
tries the branch-free form first and must leave such a solve to the plain one."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_CHILD = r"""
import time
import numpy as np
import vh
rows = vh.synthetic_eos_table()
cfg = vh.glauber_config(9, 8, 1)
cfg.dx = cfg.dy = 1e-3
cfg.dt = 0.02
cfg.etabar = 1e-35
g = np.random.default_rng(28)
e = 0.2 * 10 ** g.uniform(-3, 1, 72) + 1e-3
p = np.array([vh.eos_eval(cfg, rows, 0, v) for v in e])
u = np.zeros((4, 72))
u[0] = 1
# values too small for the branch-free form, which is computed all the same
st = vh.InitialState(e, p, u, 1e-300 * g.standard_normal((10, 72)), -1e-300 * p)
ev = vh.Event(cfg, rows)
for _ in range(2):                      # the first loads the kernels
    ev.set_initial(st)
    ev.sync()
    t = time.perf_counter()
    ev.step(1)
    ev.sync()
    t = time.perf_counter() - t
print("TIME", ev.launches_per_step(), t)
"""


def test_bisection_runs_once():
    took = {}
    for mode in ("fused", "split"):
        env = dict(os.environ, VH_STAGE_MODE=mode, PYTHONPATH=os.path.join(ROOT, "cpu-vh_b200"))
        r = subprocess.run([sys.executable, "-c", _CHILD], env=env, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        launches, t = r.stdout.split("TIME")[1].split()
        assert int(launches) == (2 if mode == "fused" else 8)
        took[mode] = float(t)
    assert took["split"] > 0.5, took            # the bisection did run on
    assert took["fused"] < 1.5 * took["split"], took
