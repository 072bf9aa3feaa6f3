"""Steps, and the allocation-free grid build, captured by the caller into a CUDA
graph of its own.  A replay finds whatever was done to the handle since: a state
set, a grid queried, plain and graphed steps; each must give the bits of the same
steps launched one by one."""
import ctypes

import numpy as np
import pytest

from arphys import FluidSim, load_library, scenes
from arphys.abi import ArpAABB

pytestmark = pytest.mark.gpu


def _scene(kind, integrator):
    if kind == "dam2d":
        return scenes.dam_break_2d(nx=24, ny=20, box=(0.5, 0.4), integrator=integrator)
    if kind == "bar3d":
        return scenes.fluid_bar_3d(fluid_n=(10, 10, 10), bar_n=(4, 12, 4), seed=3, box=(0.3, 0.2, 0.2),
                                   integrator=integrator, floor_n=(30, 20))
    sc = scenes.cantilever_bar(n=(5, 16, 5), integrator=integrator)
    for key, v in dict(plastic=1, yield_strength=100.0, relaxation_time=1e4, work_hardening_exp=2.0).items():
        sc.materials[key][1] = v
    sc.particles["vel"][:, 0] = 0.3 * np.sin(9.0 * sc.particles["pos"][:, 1])
    return sc


@pytest.mark.parametrize("kind,integrator", [("dam2d", "rk4"), ("bar3d", "rk2"), ("plastic", "rk4"),
                                             ("plastic", "verlet"), ("bar3d", "verlet")])
@pytest.mark.parametrize("before", [0, 2])
def test_a_callers_graph_of_steps_replays_like_plain_steps(kind, integrator, before):
    torch = pytest.importorskip("torch")
    if integrator == "verlet":
        before += 2  # a first step that evaluates the forces anew ends in other buffers than it began in
    sc = _scene(kind, integrator)
    sim, ref = FluidSim(sc), FluidSim(sc)
    stream = torch.cuda.Stream()
    sim.set_stream(stream.cuda_stream)
    for s in (sim, ref):
        s.init()
        s.step(before)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        sim.step(2)  # one step exchanges buffers, two end where they began

    def replay(times):
        with torch.cuda.stream(stream):
            for _ in range(times):
                graph.replay()
        ref.step(2 * times)

    def same():
        a, b = sim.particles(), ref.particles()
        assert np.isfinite(b["pos"]).all()
        assert a.tobytes() == b.tobytes()
        assert sim.solids().tobytes() == ref.solids().tobytes()

    sim.neighbors()  # a grid built between the capture and the first replay
    replay(3)
    same()
    if integrator != "verlet":  # where the graph would have to evaluate the new state's forces first
        p = ref.particles()
        p["vel"][:, 0] += 0.1
        for s in (sim, ref):
            s.set_particles(p)
        replay(2)
        same()
    for s in (sim, ref):
        s.step(2)
        s.set_graph(True)
        s.step(4)
    replay(1)
    assert sim.neighbors()["nbr_count"].tobytes() == ref.neighbors()["nbr_count"].tobytes()
    replay(1)
    same()


def test_a_callers_graph_of_the_grid_build_reads_the_positions_of_its_replay():
    torch = pytest.importorskip("torch")
    lib = load_library()
    n, h = 5000, 0.05
    bounds = ArpAABB()
    for a in range(3):
        bounds.dim[a] = 1.0
    nc = int(np.float32(1.0) / np.float32(h)) ** 3
    pos = [torch.rand((n, 4), device="cuda", generator=torch.Generator("cuda").manual_seed(q)) for q in range(2)]
    x = pos[0].clone()
    start = torch.empty(nc + 2, dtype=torch.int32, device="cuda")
    perm = torch.empty(n, dtype=torch.int32, device="cuda")

    def build():
        code = lib.arp_grid_build_noalloc(x.data_ptr(), n, ctypes.byref(bounds), float(np.float32(h)),
                                          start.data_ptr(), nc + 2, perm.data_ptr(),
                                          torch.cuda.current_stream().cuda_stream)
        assert code == 0, lib.arp_last_error()

    out = []
    for p in pos:
        x.copy_(p)
        build()
        out.append((start.clone(), perm.clone()))
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        build()
    for q in (0, 1, 0):
        x.copy_(pos[q])
        graph.replay()
        assert torch.equal(start, out[q][0]) and torch.equal(perm, out[q][1])
