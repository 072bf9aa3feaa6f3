"""The grid build's ordering and its two scatter paths where they can go wrong:
runs around the warp and block limits, more slots than a block stages, many
empty cells, and a grid of more tiles than the scatter sums up itself."""
import ctypes

import numpy as np
import pytest

from arphys import FluidSim, scenes
from arphys.abi import PARTICLE_DTYPE, ArpAABB, check, load_library

pytestmark = pytest.mark.gpu
H = np.float32(0.02)


def build(pos, cells, offset):
    """arp_grid_build_noalloc over a cube of `cells` cells a side, the cell_start
    array `offset` words past a 16-byte boundary."""
    torch = pytest.importorskip("torch")
    lib = load_library()
    n = len(pos)
    b = ArpAABB()
    box = H * np.float32(cells)
    for a in range(3):
        b.dim[a] = box
    sub = int(max(np.float32(1.0), box / H))
    nc = sub ** 3
    p = torch.zeros((max(n, 1), 4), dtype=torch.float32, device="cuda")
    p[:n, :3] = torch.from_numpy(pos).cuda()
    store = torch.full((nc + 2 + offset,), -1, dtype=torch.int32, device="cuda")
    perm = torch.full((max(n, 1),), -1, dtype=torch.int32, device="cuda")
    check(lib.arp_grid_build_noalloc(p.data_ptr(), n, ctypes.byref(b), float(H), store.data_ptr() + 4 * offset, nc + 2,
                                     perm.data_ptr(), None))
    torch.cuda.synchronize()
    return store[offset:].cpu().numpy(), perm[:n].cpu().numpy(), sub, box


@pytest.mark.parametrize("runs,offset", [([1], 0), ([32, 33, 2], 1), ([255, 256, 257], 2), ([4095, 1], 3),
                                         ([4096, 4097, 3], 0), ([20] * 230, 1)])
def test_cells_come_out_ascending_for_every_run_length(runs, offset):
    rng = np.random.default_rng(len(runs) + runs[0])
    cells = 7
    which = rng.permutation(cells ** 3)[:len(runs)]
    cell = np.repeat(which, runs)
    rng.shuffle(cell)
    xyz = np.stack([cell % cells, cell // cells % cells, cell // cells ** 2], axis=1)
    pos = ((xyz + rng.uniform(0.05, 0.95, size=xyz.shape)) * float(H)).astype(np.float32)
    bad = rng.permutation(len(pos))[:len(pos) // 10]
    pos[bad, 1] = np.nan
    start, perm, sub, box = build(pos, cells, offset)
    t = np.minimum(np.maximum(pos / box, np.float32(0)), np.float32(1))
    with np.errstate(invalid="ignore"):
        q = np.minimum(np.floor(t * np.float32(sub)), sub - 1)
    key = np.where(np.isfinite(pos).all(1), q[:, 0] + q[:, 1] * sub + q[:, 2] * sub * sub, sub ** 3).astype(np.int64)
    want = np.lexsort((np.arange(len(pos)), key))
    np.testing.assert_array_equal(perm, want)
    count = np.bincount(key, minlength=sub ** 3 + 1)
    np.testing.assert_array_equal(start, np.concatenate([[0], np.cumsum(count)]))


@pytest.mark.parametrize("box", [(0.5, 0.5, 0.5), (3.6, 3.6, 3.6)])
def test_both_scatter_paths_step_a_scene_to_the_same_state(box):
    """The same block of fluid in a small box and in one of 11.7 M search cells
    (more tiles than the scatter sums up itself).  Cells differ, so sums are
    taken in another order: equal to rounding."""
    rng = np.random.default_rng(5)
    s = 0.01
    pos = scenes.lattice((0.105,) * 3, (9, 8, 7), s) + rng.uniform(-1e-3, 1e-3, size=(504, 3))
    mats = np.array([scenes.liquid(1000.0, 20.0, 0.02, 0.1, mass=1000.0 * s ** 3)])
    p = scenes.particles(pos, 0, 1000.0 * (1 + 0.002 * rng.random(504)))
    p["vel"][:, :3] = rng.normal(0.0, 0.3, size=(504, 3))

    def run(b):
        sc = scenes.Scene(particles=p, boundary=np.zeros(0, PARTICLE_DTYPE), materials=mats,
                          bounds_min=(0.0,) * 4, bounds_dim=b + (0.0,), h=0.02, integrator="rk2", dt=1e-5)
        sim = FluidSim(sc)
        sim.init()
        sim.step(3)
        sim.set_particles(sim.particles())  # a state that replaces one already counted into cells
        sim.step(2)
        return sim.particles()
    a, b = run((0.5, 0.5, 0.5)), run(box)
    for key in ("den", "pos", "vel"):
        assert np.abs(a[key].astype(np.float64) - b[key]).max() <= 2e-6 * np.abs(a[key]).max(), key
