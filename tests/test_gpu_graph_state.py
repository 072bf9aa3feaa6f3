"""Graphed steps follow what the host changes between them."""
import numpy as np
import pytest

from arphys import FluidSim, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("integrator", ["rk2", "verlet"])
@pytest.mark.parametrize("first", [1, 2])  # steps before the change: either set of buffers
def test_graphed_steps_after_the_stiffness_is_cleared_read_the_materials(first, integrator):
    sc = scenes.cantilever_bar(n=(5, 16, 5), integrator=integrator)
    sc.particles["vel"][:, 0] = 0.3 * np.sin(9.0 * sc.particles["pos"][:, 1])
    out = []
    for graph in (False, True):
        sim = FluidSim(sc)
        sim.init()
        sim.set_graph(graph)
        sim.step(4)  # both sets of buffers are captured with the materials' stiffness
        sim.set_solid_stiffness(5.0 * np.asarray(sc.meta["stiffness"], np.float32))
        sim.step(first)
        sim.set_solid_stiffness(None)
        sim.step(3)
        out.append(sim.particles())
    assert np.isfinite(out[0]["pos"]).all()
    assert out[0].tobytes() == out[1].tobytes()


@pytest.mark.parametrize("integrator", ["rk2", "verlet"])
def test_graphed_steps_after_a_second_init_run_from_the_initial_state(integrator):
    sc = scenes.cantilever_bar(n=(5, 16, 5), integrator=integrator)
    sc.particles["vel"][:, 0] = 0.3 * np.sin(9.0 * sc.particles["pos"][:, 1])
    out = []
    for graph in (False, True):
        sim = FluidSim(sc)
        sim.init()
        sim.set_graph(graph)
        sim.step(5)
        sim.init()
        other = FluidSim(scenes.cantilever_bar(n=(6, 20, 6)))  # takes memory that the second init has given back
        other.init()
        sim.step(5)
        out.append(sim.particles())
    assert np.isfinite(out[0]["pos"]).all()
    assert out[0].tobytes() == out[1].tobytes()
