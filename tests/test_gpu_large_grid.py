"""Grids of more cells than one scan's tile totals cover, few of them occupied: the
occupancy counters, which such a grid's blocks take for their own cells, and the
step against the oracle."""
import numpy as np
import pytest

from arphys import FluidSim, scenes
from arphys.abi import PARTICLE_DTYPE
from helpers import rel_err
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


# cells along x: one grid below and one above 8,192 blocks of 256 search cells, one past 4 M search cells
@pytest.mark.parametrize("cells", [(100, 100, 100), (150, 100, 100), (250, 100, 100)])
def test_occupancy_counters_and_steps_of_a_large_sparse_grid(cells):
    rng = np.random.default_rng(sum(cells))
    h = 0.01
    side = [h * (c + 0.25) for c in cells]
    clusters = rng.uniform(0.1, 0.9, size=(40, 3)) * side
    pos = np.concatenate([c + rng.uniform(-0.7 * h, 0.7 * h, size=(60, 3)) for c in clusters])
    pos[:150] = (np.array([30, 20, 10]) + rng.uniform(0.2, 0.8, size=(150, 3))) * np.array(side) / cells  # one cell
    mats = np.array([scenes.liquid(1000.0, 20.0, h, 0.1, mass=1000.0 * (0.3 * h) ** 3)])
    p = scenes.particles(pos, 0, 1000.0 * (1.0 + 0.01 * rng.random(len(pos))))
    p["vel"][:, :3] = rng.normal(0.0, 0.5, size=(len(pos), 3))
    sc = scenes.Scene(particles=p, boundary=np.zeros(0, PARTICLE_DTYPE), materials=mats, bounds_min=(0.0,) * 4,
                      bounds_dim=tuple(side) + (0.0,), h=h, integrator="rk2", dt=1e-6, gravity=0.0, name="sparse")
    sim = FluidSim(sc)
    sim.init()
    f = np.float32
    key = np.zeros(len(p), np.int64)
    for a in (2, 1, 0):
        t = np.clip((p["pos"][:, a] - f(0.0)) / f(side[a]), f(0), f(1)) * f(cells[a])
        key = key * cells[a] + np.minimum(np.floor(t).astype(np.int64), cells[a] - 1)
    occ = np.bincount(key)
    assert occ.max() == 150 and (occ > 128).sum() == 1
    for graph in (False, True):
        sim.set_graph(graph)
        sim.set_particles(p)
        sim.step(2)
    st = sim.stats()
    assert st["max_cell_occupancy"] == 150 and st["nonfinite_positions"] == 0
    assert st["overflow_cells"] == 2 * 2 * 2  # once a stage
    # away from the crowded cell, which the oracle's buckets cut off at 128
    far = np.abs(pos - pos[:150].mean(axis=0)).max(axis=1) > 4 * h
    assert far.sum() > 1000
    o = Oracle(sc, 64)
    o.step(2)
    r, got = o.state(), sim.particles()
    for k in ("den", "vel"):
        assert rel_err(got[k][far], r[k][far]) < 1e-5, k
