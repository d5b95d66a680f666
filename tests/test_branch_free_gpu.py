"""The branch-free flux, source and inversion (vh_math.cuh, vh_physics.cuh,
vh_stage.cuh) where they can go wrong, bit for bit against the oracle: lattices
at the edges of the line pieces and of the fused/split rule, and states whose
values leave the range the quotients are exact in, so that cells, blocks or
single quotients fall back to the plain operations."""
import os
import sys

import numpy as np
import pytest

import vh

pytestmark = pytest.mark.gpu
sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "oracle"))
from oracle import OracleEvent  # noqa: E402

FIELDS = list(range(15)) + [100, 101, 102, 103, 200, 201]


def state(cfg, scale, seed=3):
    """a smooth event with flow; pi, Pi and the flow along one axis of magnitude scale"""
    rng = np.random.default_rng(seed)
    rows = vh.synthetic_eos_table()
    x = [(np.arange(n) - (n - 1) / 2) for n in (cfg.nx, cfg.ny, cfg.nz)]
    z, y, x = np.meshgrid(x[2] * cfg.dz, x[1] * cfg.dy, x[0] * cfg.dx, indexing="ij")
    e = 25.0 * np.exp(-(x ** 2 + y ** 2) / 18 - z ** 2 / 8) * (1 + 0.1 * np.sin(x + y)) + 2e-3
    e = e.reshape(-1)
    p = np.array([vh.eos_eval(cfg, rows, 0, v) for v in e])
    ux, uy, un = 0.1 * np.tanh(x / 4).reshape(-1), scale * np.sin(y).reshape(-1), np.zeros(e.size)
    u = np.stack([np.sqrt(1 + ux ** 2 + uy ** 2), ux, uy, un])
    pi = scale * rng.standard_normal((10, e.size)) * e
    pi[:, ::7] = 0.0
    pi[2, ::5] = -0.0
    return rows, vh.InitialState(e, p, u, pi, -scale * p)


def same_bits(cfg, rows, st, steps):
    gpu, orc = vh.Event(cfg, rows), OracleEvent(cfg, rows)
    gpu.set_initial(st)
    orc.set_initial(st)
    gpu.step(steps)
    assert orc.step(steps) == 0
    gpu.sync()
    bad = {}
    for f in FIELDS:
        a, b = vh.face_cells(cfg, gpu.field(f)), vh.face_cells(cfg, orc.field(f))
        n = int(np.count_nonzero(a.view(np.uint64) != b.view(np.uint64)))
        if n:
            bad[f] = n
    launches = gpu.launches_per_step()
    gpu.close()
    assert not bad, f"bit-differing cells per field: {bad}"
    return launches


@pytest.mark.parametrize("size, launches", [
    ((33, 19, 9), 10),        # two bundles of rows, a ragged last column
    ((35, 61, 3), 10),        # eta lines of 3 cells: twelve pieces in a block
    ((37, 80, 2), 10),        # of 2: a piece's first two threads are its last two
    ((2, 160, 3), 10),        # x lines of 2
    ((160, 2, 31), 10),       # y lines of 2
    ((32, 16, 18), 2),        # 288 blocks
    ((32, 16, 20), 10),       # 320, and no ragged end
    ((31, 148, 2), 2),        # the fused form's largest 3+1D grid, 296 blocks
    ((31, 149, 2), 10),
    ((64, 222, 1), 2),        # and 2+1D, 444
    ((64, 223, 1), 8),
])
def test_lattice_edges(size, launches):
    cfg = vh.glauber_config(*size)
    cfg.dx = cfg.dy = 0.3
    rows, st = state(cfg, 1e-2)
    assert same_bits(cfg, rows, st, 2) == launches


@pytest.mark.parametrize("scale", [0.0, 1e-30, 1e-44, 1e-47, 1e-80, 1e-150, 1e-290, 1e-308, 1e-320])
@pytest.mark.parametrize("size", [(33, 19, 9), (21, 17, 1)])
def test_values_out_of_range(size, scale):
    cfg = vh.glauber_config(*size)
    cfg.dx = cfg.dy = 0.3
    rows, st = state(cfg, scale)
    same_bits(cfg, rows, st, 2)
