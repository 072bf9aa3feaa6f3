"""The solid kernels share a solid between 4 threads below a number of solids
and 2 above it; both add the same partial sums, so a scene gives the same bits
alone and in a batch that passes the line."""
import numpy as np
import pytest

from arphys import FluidSim, scenes

pytestmark = pytest.mark.gpu

FEW = 24576  # csrc/solid.cu: kFewSolids


@pytest.mark.parametrize("order,plastic", [(2, False), (2, True), (0, False)])
def test_a_solid_scene_gives_the_same_bits_with_either_number_of_threads(order, plastic):
    def bar(n, seed):
        sc = scenes.cantilever_bar(n=n, seed=seed, v_sigma=0.5)
        sc.materials["strain_order"][1] = order
        if plastic:
            for key, v in dict(plastic=1, yield_strength=50.0, relaxation_time=1e4, work_hardening_exp=2.0).items():
                sc.materials[key][1] = v
        return sc
    small = [bar((2, 5, 2), 1), bar((3, 7, 5), 2)]
    big = bar((16, 120, 14), 3)
    assert sum(sc.n for sc in small) <= FEW < big.n
    batch = FluidSim.batch(small + [big])
    batch.init()
    batch.step(3)
    p, s = batch.particles(), batch.solids()
    first_solid = 0
    for k, sc in enumerate(small):
        sim = FluidSim(sc)
        sim.init()
        sim.step(3)
        first, n = batch.scene_range(k)[:2]
        assert np.isfinite(sim.particles()["pos"]).all()
        assert p[first:first + n].tobytes() == sim.particles().tobytes(), k
        assert s["stress"][first_solid:first_solid + sim.ns].tobytes() == sim.solids()["stress"].tobytes(), k
        first_solid += sim.ns
