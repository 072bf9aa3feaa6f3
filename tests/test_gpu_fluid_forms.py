"""The fluid kernel's forms where they can go wrong: particle counts around a
warp, a block and a group, grids of one to three cells (where quantised
positions wrap), walls, contact and friction, and the scan's integer test
itself (on the CPU, against the distances it stands for)."""
import numpy as np
import pytest

from arphys import FluidSim, scenes
from arphys.abi import CONTACT_LINEAR, INTERACTION_DTYPE, PARTICLE_DTYPE
from helpers import rel_err
from oracle.oracle import Oracle

UNITS, BOUND = 63.0, 4273


def block(n, dim, cells, seed, wall=False):
    """`n` fluid particles at random lattice sites of a box of `cells` cells of
    1.9 h a side (so cells are wide and differences exceed 2 h), a second
    fluid in contact with the first among them, optionally a wall layer (contact
    and friction)."""
    rng = np.random.default_rng(seed)
    h = 0.02
    side = 1.9 * h * cells
    m = int(np.ceil(n ** (1.0 / dim))) + 1
    s = side / m
    pos = scenes.lattice((0.5 * s,) * dim, (m,) * dim, s)
    pos = pos[rng.permutation(len(pos))[:n]]
    pos = pos + rng.uniform(-0.2 * s, 0.2 * s, size=pos.shape)
    mass = 1000.0 * s ** dim
    mats = np.array([scenes.immobile(0.3, mass=s ** dim), scenes.liquid(1000.0, 20.0, h, 0.1, visc=0.5, mass=mass),
                     scenes.liquid(1100.0, 15.0, h, 0.2, mass=mass)])
    inter = np.zeros((3, 3), INTERACTION_DTYPE)
    given = np.zeros((3, 3), np.uint8)
    inter[1, 2] = (CONTACT_LINEAR, 5000.0, 0.03, 0.1, 0.0)  # potential, strength, radius, dampening, friction
    given[1, 2] = 1
    mat = np.where(rng.random(n) < 0.2, 2, 1).astype(np.uint32)
    p = scenes.particles(pos, mat, np.where(mat == 2, 1100.0, 1000.0) * (1 + 0.01 * rng.random(n)))
    p["vel"][:, :dim] = rng.normal(0.0, 0.5, size=(n, dim))
    b = np.zeros(0, PARTICLE_DTYPE)
    if wall:
        w = scenes.lattice((0.5 * s,) * dim, (m,) * (dim - 1) + (1,), s)
        w[:, dim - 1] = -0.5 * s
        b = scenes.particles(w, 0, 1.0)
    return scenes.Scene(particles=p, boundary=b, materials=mats, bounds_min=(0.0,) * 4,
                        bounds_dim=tuple([side] * dim + [0.0] * (4 - dim)), h=h, integrator="rk2", dt=1e-5,
                        gravity=9.81, interactions=inter, interaction_given=given, name=f"block_{n}_{dim}d_{cells}")


@pytest.mark.gpu
@pytest.mark.parametrize("n,dim,cells,wall", [(1, 3, 1, False), (2, 2, 1, True), (31, 2, 1, True), (33, 3, 1, True),
                                              (127, 3, 2, True), (129, 2, 2, False), (257, 3, 2, True),
                                              (1000, 3, 3, True)])
def test_every_form_gives_the_same_bits_and_the_oracles_result(n, dim, cells, wall):
    sc = block(n, dim, cells, seed=n, wall=wall)
    ref = None
    for v in range(FluidSim.fluid_variant_count()):
        sim = FluidSim(sc)
        sim.init()
        sim.set_fluid_variant(v)
        sim.step(3)
        p = sim.particles()
        ref = p if ref is None else ref
        assert p.tobytes() == ref.tobytes(), v
    o = Oracle(sc, 64)
    o.step(3)
    r = o.state()
    o32 = Oracle(sc, 32)
    o32.step(3)
    r32 = o32.state()
    for key in ("den", "pos", "vel"):
        # as close to the double oracle as twice the float oracle is, or 1e-6
        assert rel_err(ref[key], r[key]) <= max(1e-6, 2.0 * rel_err(r32[key], r[key])), key


@pytest.mark.gpu
def test_cells_counted_with_the_state_follow_every_change_of_it():
    """A step leaves its last state counted into cells for the next; a state set
    or queried in between, or a profiled step, must not see stale cells."""
    sc = block(300, 3, 3, seed=7, wall=True)
    a, b = FluidSim(sc), FluidSim(sc)
    for sim in (a, b):
        sim.init()
    a.step(4)
    b.step(2)
    mid = b.particles()
    b.set_graph(True)
    b.neighbors()  # builds another grid in the same buffers
    b.step(1)
    b.set_particles(mid)
    b.profile_enable(True)
    b.step(1)
    b.profile_enable(False)
    b.step(1)
    assert a.particles().tobytes() == b.particles().tobytes()
    assert a.stats() != {} and a.stats()["nonfinite_positions"] == 0


@pytest.mark.parametrize("h,extent", [(0.02, 2.56), (0.013, 40.0), (3.0, 7.0)])
def test_quantised_scan_lets_every_pair_within_h_through(h, extent):
    """The scan's integer test restated: no pair within h fails it, and the test
    lets through at most the pairs within 1.08 h (differences below the wrap)."""
    rng = np.random.default_rng(3)
    h32 = float(np.float32(h))
    a = rng.uniform(0.0, extent, size=(200000, 3)).astype(np.float32).astype(np.float64)
    d = rng.normal(size=a.shape)
    d *= (h32 * rng.uniform(0.9, 1.2, size=(len(a), 1))) / np.linalg.norm(d, axis=1, keepdims=True)
    b = (a + d).astype(np.float32).astype(np.float64)
    inv = UNITS / h32

    def code(p, shift):
        q = np.rint(p * inv - np.array([0.0, shift, shift])).astype(np.int64) & 255
        return q[:, 0] | q[:, 1] << 8 | q[:, 2] << 16
    diff = ((code(b, 0.0) - code(a, 0.5)) & 0xFFFFFFFF).astype(np.uint32)
    by = np.stack([(diff >> (8 * k) & 255).astype(np.uint8).view(np.int8).astype(np.int64) for k in range(4)])
    passed = (by ** 2).sum(0) <= BOUND
    r = np.linalg.norm(b - a, axis=1)
    assert passed[r < h32].all()
    assert not passed[r > 1.08 * h32].any()
