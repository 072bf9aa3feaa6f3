"""The fluid kernel runs beside the solid kernels and waits for them in its
epilogue.  Plain launches, graph replay and profiled steps (whose timing events
lie between the kernels) give the same bits."""
import numpy as np
import pytest

from arphys import FluidSim, scenes

pytestmark = pytest.mark.gpu


def _scene(f, b, integrator):
    box = (round(0.01 * (f + b + 16), 6), round(0.01 * max(f + 8, 4 * b + 4), 6), round(0.01 * (max(f, b) + 8), 6))
    return scenes.fluid_bar_3d(fluid_n=(f, f, f), bar_n=(b, 4 * b, b), seed=3, box=box, integrator=integrator,
                               floor_n=(int(round(box[0] * 100)), int(round(box[2] * 100))))


# solids: less than a block of the solid kernels, less than a wave of them, more than one wave
@pytest.mark.parametrize("f,b", [(6, 2), (12, 9), (40, 22)])
@pytest.mark.parametrize("integrator", ["rk4", "verlet"])
def test_plain_graphed_and_profiled_steps_with_solids_give_the_same_bits(f, b, integrator):
    out = []
    for mode in ("plain", "graph", "profiled"):
        for variant in (2, 13):  # the block form and the group form
            sim = FluidSim(_scene(f, b, integrator))
            sim.init()
            sim.set_fluid_variant(variant)
            sim.set_graph(mode == "graph")
            if mode == "profiled":
                sim.profile_enable()
            sim.step(6)
            out.append(sim.particles().tobytes())
            if mode == "profiled":
                assert sim.profile_read()["solid_launches"] > 0
            assert np.isfinite(sim.particles()["pos"]).all()
            sim.close()
    assert all(o == out[0] for o in out[1:])
