"""What a step carries over to the next (the state counted into cells; for velocity
Verlet the kicked and drifted state and the kicked plastic strain) survives or is
made anew whatever is asked of the handle in between; and the pairs that the
kernel's quantised scan lists."""
import numpy as np
import pytest

from arphys import FluidSim, scenes
from arphys.abi import PARTICLE_DTYPE
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _scene(kind, integrator):
    if kind == "bar3d":
        sc = scenes.fluid_bar_3d(fluid_n=(10, 10, 10), bar_n=(4, 12, 4), seed=3, box=(0.3, 0.2, 0.2),
                                 integrator=integrator, floor_n=(30, 20))
    else:
        sc = scenes.cantilever_bar(n=(5, 16, 5), integrator=integrator)
        for key, v in dict(plastic=1, yield_strength=100.0, relaxation_time=1e4, work_hardening_exp=2.0).items():
            sc.materials[key][1] = v
    sc.particles["vel"][:, 0] += 0.3 * np.sin(9.0 * sc.particles["pos"][:, 1]).astype(np.float32)
    return sc


BETWEEN = {"neighbors": lambda s: s.neighbors(), "autotune": lambda s: s.autotune(),
           "device_state": lambda s: s.device_state(), "particles": lambda s: s.particles(),
           "solids": lambda s: s.solids(), "stats": lambda s: s.stats(),
           "boundary_cells": lambda s: s.boundary_cells()}


@pytest.mark.parametrize("what", sorted(BETWEEN))
@pytest.mark.parametrize("kind,integrator", [("plastic", "verlet"), ("plastic", "rk4"), ("bar3d", "verlet")])
def test_steps_are_the_same_whatever_is_asked_between_them(kind, integrator, what):
    sc = _scene(kind, integrator)
    a, b = FluidSim(sc), FluidSim(sc)
    for sim in (a, b):
        sim.init()
    a.step(8)
    b.step(2)
    BETWEEN[what](b)
    b.step(1)
    BETWEEN[what](b)
    b.set_graph(True)
    b.step(2)
    BETWEEN[what](b)
    b.step(1)  # a graphed step that finds its state uncounted
    b.profile_enable(True)
    b.step(1)
    b.profile_enable(False)
    BETWEEN[what](b)
    b.set_graph(False)
    b.step(1)
    assert np.isfinite(a.particles()["pos"]).all()
    assert a.particles().tobytes() == b.particles().tobytes()
    assert a.solids().tobytes() == b.solids().tobytes()


@pytest.mark.parametrize("variant", [0, 14])  # the block form and the group form
@pytest.mark.parametrize("dim", [2, 3])
def test_pairs_just_inside_h_are_found_at_every_phase_of_the_codes(variant, dim):
    """Isolated pairs a hair inside h, their first particle at every phase of the
    8-bit codes (steps of 1/63 h over 256 of them, offset by fractions of a step, so
    differences wrap and borrow), along the axes and the diagonals that carry the
    bound.  A pair that the scan lost would have no density rate; the others' are
    the oracle's."""
    rng = np.random.default_rng(11)
    h = 0.02
    n_pairs = 4096 if dim == 3 else 1024
    per = int(round(n_pairs ** (1.0 / dim)))
    pitch = 3.3 * h  # pairs are out of one another's reach
    grid = np.stack(np.meshgrid(*[np.arange(per)] * dim, indexing="ij"), -1).reshape(-1, dim)
    a = 1.5 * h + pitch * grid + h / 63.0 * (rng.integers(0, 8, grid.shape) + rng.choice([0.0, 0.25, 0.49, 0.5, 0.51, 0.75],
                                                                                       grid.shape))
    d = rng.choice([-1.0, 0.0, 1.0], size=grid.shape)
    d[~d.any(axis=1), 0] = 1.0
    d += 0.02 * rng.normal(size=d.shape) * rng.integers(0, 2, size=(len(d), 1))
    d *= (h * rng.choice([0.9, 0.98, 0.995], size=(len(d), 1))) / np.linalg.norm(d, axis=1, keepdims=True)
    pos = np.concatenate([a, a + d])
    side = 3.0 * h + pitch * per
    mats = np.array([scenes.liquid(1000.0, 20.0, h, 0.1, mass=1000.0 * (0.5 * h) ** dim)])
    p = scenes.particles(pos, 0, 1000.0)
    p["vel"][:, :dim] = np.concatenate([np.zeros_like(d), d / h])  # drifting apart
    sc = scenes.Scene(particles=p, boundary=np.zeros(0, PARTICLE_DTYPE), materials=mats, bounds_min=(0.0,) * 4,
                      bounds_dim=tuple([side] * dim + [0.0] * (4 - dim)), h=h, integrator="euler", dt=1e-3,
                      gravity=0.0, name="pairs")
    r = np.linalg.norm(p["pos"][len(a):, :dim].astype(np.float64) - p["pos"][:len(a), :dim].astype(np.float64), axis=1)
    assert (r < np.float32(h)).all() and (r > 0.85 * h).all()
    sim = FluidSim(sc)
    sim.init()
    sim.set_fluid_variant(variant)
    sim.step(1)
    o = Oracle(sc, 64)
    o.step(1)
    got, want = sim.particles()["den"].astype(np.float64) - 1000.0, o.state()["den"] - 1000.0
    assert (want < 0).all()
    # one float32 rounding of a density near 1000, and of the pair's term
    assert np.abs(got - want).max() <= 2.0 ** -14 + 1e-5 * np.abs(want).max(), np.abs(got - want).max()
    assert np.abs(want).min() > 8 * 2.0 ** -14  # a lost pair would show
