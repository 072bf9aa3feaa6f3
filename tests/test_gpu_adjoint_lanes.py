"""The reverse pass shares a particle or a solid between 8 threads below a
number of them and 2 above it; a scene's gradients are the same either way, up
to the order of the sums."""
import numpy as np
import pytest

from arphys import FluidSim, scenes

pytestmark = pytest.mark.gpu

FEW, FEW_SOLIDS = 24576, 16384  # csrc/adjoint.cu: kAdjFew, kAdjFewSolids


def bars(sizes):
    return [scenes.fluid_bar_3d(fluid_n=f, bar_n=b, floor_n=w, seed=k) for k, (f, b, w) in enumerate(sizes)]


def dams(sizes):
    return [scenes.dam_break_2d(nx=nx, ny=ny, seed=k) for k, (nx, ny) in enumerate(sizes)]


@pytest.mark.parametrize("make,sizes", [
    (bars, [((2, 5, 3), (2, 4, 2), (12, 12)), ((9, 7, 5), (3, 8, 3), (20, 16)), ((21, 20, 20), (20, 42, 22), (64, 64))]),
    (dams, [(1, 1), (3, 5), (37, 23), (256, 128)])])
def test_a_scene_has_the_same_gradients_with_either_number_of_threads(make, sizes):
    scs = make(sizes)
    small, big = scs[:-1], scs[-1]
    assert sum(sc.n for sc in small) <= FEW < big.n
    if make is bars:
        assert sizes[-1][1][0] * (sizes[-1][1][1] - 2) * sizes[-1][1][2] > FEW_SOLIDS
    rng = np.random.default_rng(9)
    dim = 3 if make is bars else 2
    gs = []
    for sc in scs:
        sc.particles["vel"][:, :dim] = rng.normal(0.0, 0.2, size=(sc.n, dim)).astype(np.float32)
        g = np.zeros((sc.n, 8), np.float32)
        g[:, :dim] = rng.normal(size=(sc.n, dim))
        gs.append(g)

    def gradients(sim, g):
        sim.init()
        sim.tape_begin(2)
        sim.step(3)
        out = sim.backward(g)[0]
        sim.tape_end()
        return out
    batch = FluidSim.batch(scs)
    gb = gradients(batch, np.concatenate(gs))
    off = np.cumsum([0] + [sc.n for sc in scs])
    assert np.isfinite(gb).all()
    for k, sc in enumerate(small):
        g = gradients(FluidSim(sc), gs[k])
        # sums of up to some sixty float terms, at most a few times larger than
        # their result in the norm: 60 * 2^-24 * 3
        err = np.linalg.norm(gb[off[k]:off[k + 1]] - g) / np.linalg.norm(g)
        print(f"scene {k}: {err:.1e}")
        assert err < 1e-5, k
