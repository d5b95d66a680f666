"""2+1D freezeout blocks where Cornelius has its hard cases: cell-scale noise
around the freezeout energy density, some corners exactly on it, so that cubes
are ambiguous and have up to four elements; and surfaces on either side of the
512 elements that are also kept in pinned memory.  Every element bit for bit
against the oracle, from the count step's slots and, with room for one element
only, computed again by one thread per cube."""
import numpy as np
import pytest

import vh
from oracle import OracleEvent

pytestmark = pytest.mark.gpu


def conformal_state(cfg, e, u_perp):
    u = np.stack([np.sqrt(1 + u_perp[0] ** 2 + u_perp[1] ** 2), u_perp[0], u_perp[1], np.zeros(e.size)])
    return vh.InitialState(e, e / 3, u, np.zeros((10, e.size)), None)


def block(gpu, orc):
    n, above = gpu.freezeout()
    got = gpu.surface()
    want, above_o = orc.freezeout()
    assert (n, above) == (len(want), above_o)
    np.testing.assert_array_equal(got.view(np.uint64), want.view(np.uint64))
    return want


@pytest.mark.parametrize("initial_cap", [None, "1"])
def test_noise(initial_cap, monkeypatch):
    if initial_cap:
        monkeypatch.setenv("VH_FO_INITIAL_CAP", initial_cap)
    cfg = vh.gubser_config(61, 53)
    cfg.dx = cfg.dy = 0.25
    cfg.dt, cfg.fo_factor, cfg.T_freezeout_GeV = 0.1, 5, 0.2
    gpu, orc = vh.Event(cfg), OracleEvent(cfg)
    eF = orc.L.vho_fo_eF(orc.h)
    per_cube = np.zeros(5, int)
    for seed in (1, 2, 3):
        rng = np.random.default_rng(seed)
        N = cfg.nx * cfg.ny
        e = eF * np.exp(rng.uniform(-1, 1, N))
        e[rng.random(N) < 0.1] = eF
        st = conformal_state(cfg, e, 0.3 * rng.standard_normal((2, N)))
        gpu.set_initial(st)
        orc.set_initial(st)
        block(gpu, orc)
        gpu.step(cfg.fo_factor)
        assert orc.step(cfg.fo_factor) == 0
        rows = block(gpu, orc)
        ix = np.floor(rows[:, 1] / cfg.dx + (cfg.nx - 1) / 2).astype(int)
        iy = np.floor(rows[:, 2] / cfg.dy + (cfg.ny - 1) / 2).astype(int)
        per_cube += np.bincount(np.bincount(ix * cfg.ny + iy), minlength=5)
    assert per_cube[1] > 1000 and per_cube[2] > 1000 and per_cube[3] > 10 and per_cube[4] > 0, per_cube


@pytest.mark.parametrize("initial_cap", [None, "600"])
@pytest.mark.parametrize("lone, corner, elements", [(127, 3, 511), (128, 0, 512), (128, 1, 513), (129, 0, 516)])
def test_pinned_rows_edge(lone, corner, elements, initial_cap, monkeypatch):
    """cells above e_F with none around them: four elements each against the
    first block's zero slab, one where the cell is a corner of the lattice"""
    if initial_cap:
        monkeypatch.setenv("VH_FO_INITIAL_CAP", initial_cap)
    cfg = vh.gubser_config(61, 61)
    gpu, orc = vh.Event(cfg), OracleEvent(cfg)
    eF = orc.L.vho_fo_eF(orc.h)
    e = np.full((61, 61), 0.5 * eF)
    spots = [(y, x) for y in range(3, 58, 3) for x in range(3, 58, 3)][:lone]
    for y, x in spots + [(0, 0), (0, 60), (60, 0)][:corner]:
        e[y, x] = 2 * eF
    st = conformal_state(cfg, e.reshape(-1), np.zeros((2, 61 * 61)))
    gpu.set_initial(st)
    orc.set_initial(st)
    assert len(block(gpu, orc)) == elements
    gpu.step(1)
    assert orc.step(1) == 0
    block(gpu, orc)
