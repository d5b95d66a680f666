"""Values of theta at which the branch-free limiter (vh_physics.cuh, limited)
does not hold: bit for bit against the oracle on fused and phase-split lattices
and in a batch."""
import numpy as np
import pytest

import vh
from oracle import OracleEvent

pytestmark = pytest.mark.gpu
FIELDS = list(range(15)) + [100, 101, 102, 103, 200, 201]
SIZES = [(21, 17, 1), (33, 19, 9), (64, 223, 1)]        # fused 2+1D, split 3+1D, split 2+1D
SPLIT = {(21, 17, 1): 2, (33, 19, 9): 10, (64, 223, 1): 8}


def event_state(size):
    cfg = vh.glauber_config(*size)
    cfg.dx = cfg.dy = 0.3
    rows = vh.synthetic_eos_table()
    rng = np.random.default_rng(5)
    z, y, x = np.meshgrid(*[(np.arange(n) - (n - 1) / 2) * d for n, d in
                            ((cfg.nz, cfg.dz), (cfg.ny, cfg.dy), (cfg.nx, cfg.dx))], indexing="ij")
    e = (25.0 * np.exp(-(x ** 2 + y ** 2) / 18 - z ** 2 / 8) * (1 + 0.1 * np.sin(x + y)) + 2e-3).reshape(-1)
    p = np.array([vh.eos_eval(cfg, rows, 0, v) for v in e])
    ux, uy, un = 0.1 * np.tanh(x / 4).reshape(-1), 0.05 * np.sin(y).reshape(-1), np.zeros(e.size)
    u = np.stack([np.sqrt(1 + ux ** 2 + uy ** 2), ux, uy, un])
    pi = 1e-2 * rng.standard_normal((10, e.size)) * e
    pi[:, ::7] = 0.0
    return cfg, rows, vh.InitialState(e, p, u, pi, -1e-2 * p)


def compare(cfg, gpu, orc):
    bad = {}
    for f in FIELDS:
        a, b = vh.face_cells(cfg, gpu.field(f)), vh.face_cells(cfg, orc.field(f))
        n = int(np.count_nonzero(a.view(np.uint64) != b.view(np.uint64)))
        if n:
            bad[f] = n
    assert not bad, f"differing cells per field: {bad}"


def run(cfg, rows, st, steps, batch=False):
    gpu, orc = vh.Event(cfg, rows), OracleEvent(cfg, rows)
    gpu.set_initial(st)
    orc.set_initial(st)
    if batch:
        vh.Batch([gpu]).step(steps)
    else:
        gpu.step(steps)
    assert orc.step(steps) == 0
    gpu.sync()
    return gpu, orc


@pytest.mark.parametrize("theta", [np.inf, -np.inf, np.nan, 0.0, -1.8, 1e-30, 1e-250, 1e300])
@pytest.mark.parametrize("size", SIZES)
def test_theta(size, theta):
    cfg, rows, st = event_state(size)
    cfg.theta = theta
    gpu, orc = run(cfg, rows, st, 2)
    assert gpu.launches_per_step() == SPLIT[size]
    compare(cfg, gpu, orc)
    gpu.close()


@pytest.mark.parametrize("size", SIZES[:2])
def test_batch(size):
    cfg, rows, st = event_state(size)
    cfg.theta = np.inf
    gpu, orc = run(cfg, rows, st, 2, batch=True)
    compare(cfg, gpu, orc)
    gpu.close()
