"""A scene that is flat in z when it is created is stepped and differentiated in
the plane, whatever z and vz a state set later holds: distances, and so densities,
forces and gradients, are those of the same particles with z = 0."""
import numpy as np
import pytest

from arphys import FluidSim, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 9, 12, 13, 14])  # both forms of the fluid kernel
@pytest.mark.parametrize("integrator", ["rk2", "verlet"])
def test_a_flat_scene_ignores_z(variant, integrator):
    sc = scenes.dam_break_2d(nx=40, ny=30, box=(0.8, 0.5), integrator=integrator)
    rng = np.random.default_rng(5)
    flat = sc.particles.copy()
    flat["vel"][:, :2] = rng.normal(0.0, 0.5, size=(sc.n, 2))
    off = flat.copy()
    # a fraction of h, where only pairs close to h apart would be lost, up to where 8-bit codes wrap
    off["pos"][:, 2] = sc.h * rng.uniform(0.0, 1.0, sc.n) * rng.choice([0.5, 3.0, 9.0], sc.n)
    off["vel"][:, 2] = rng.normal(0.0, 1.0, sc.n)
    dl = rng.normal(size=(sc.n, 8)).astype(np.float32)
    dl[:, [2, 6, 7]] = 0.0
    states, grads = [], []
    for p in (flat, off):
        sim = FluidSim(sc)
        sim.init()
        sim.set_fluid_variant(variant)
        sim.set_particles(p)
        sim.step(3)
        sim.tape_begin(1)
        sim.step(2)
        states.append(sim.particles())
        grads.append(sim.backward(dl)[0])
        sim.tape_end()
    a, b = states
    assert np.isfinite(b["pos"]).all()
    for key, cols in (("den", Ellipsis), ("pos", (slice(None), [0, 1])), ("vel", (slice(None), [0, 1]))):
        assert np.array_equal(a[key][cols], b[key][cols]), key
    np.testing.assert_array_equal(b["vel"][:, 2], off["vel"][:, 2])  # nothing acts along z
    assert np.abs(grads[0]).max() > 0
    assert np.array_equal(grads[0], grads[1])


def test_a_batch_of_flat_scenes_ignores_z():
    scs = [scenes.dam_break_2d(nx=n, ny=20, box=(0.5, 0.4), seed=n) for n in (20, 23)]
    out = []
    for z in (0.0, 1.0):
        sim = FluidSim.batch(scs)
        sim.init()
        p = sim.particles()
        p["pos"][:, 2] = z * np.random.default_rng(2).uniform(0.0, 0.1, len(p))
        sim.set_particles(p)
        sim.step(4)
        out.append(sim.particles())
    assert np.array_equal(out[0]["den"], out[1]["den"])
    assert np.array_equal(out[0]["vel"], out[1]["vel"])
    assert np.array_equal(out[0]["pos"][:, :2], out[1]["pos"][:, :2])
