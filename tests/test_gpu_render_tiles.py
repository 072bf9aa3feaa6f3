"""Splat compositing where it can go wrong: tiles with the sprites of several
draw-order chunks, tiles cut by the frame's edge, sprites larger than a tile,
frames of one pixel, byte for byte against the oracle; and the blend's
divisions by constants."""
import numpy as np
import pytest

from arphys import FluidSim, scenes
from oracle.oracle import norm_const_f32
from test_gpu_render import oracle_frame, style_for


def test_the_blend_divides_by_its_constants_exactly():
    """q / 255 and wk / kconst as x hi + x lo, hi + lo the constant's reciprocal
    in two floats, over every value they are used for (csrc/renderer.cu)."""
    def check(x, const, hi, lo):
        y = x.astype(np.float64) * np.float64(hi) + (x * lo).astype(np.float64)  # the first product is exact
        assert not np.any((y.view(np.uint64) & 0x1FFFFFFF) == 0x10000000)  # so rounding twice is rounding once
        assert (y.astype(np.float32) == x / const).all()

    f = np.float32
    check(np.arange(256).astype(f), f(255), f(float.fromhex("0x1.010102p-8")), f(float.fromhex("-0x1.fdfdfep-33")))
    k = f(norm_const_f32(3, 3.0))
    hi = f(1) / k
    d = (np.arange(2 ** 24 + 1) / 2.0 ** 24).astype(f)
    check(((k * d) * d) * d, k, hi, f(1.0 / float(k) - float(hi)))


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,nx,ny,size,scale", [
    (1, 1, 40, 40, 4.0, 1.45), (17, 33, 60, 60, 4.0, 1.45), (16, 16, 48, 32, 30.0, 1.45), (70, 50, 64, 64, 1.0, 1.2),
    (48, 80, 33, 31, 60.0, 1.4)])
def test_splat_tiles_of_several_chunks_match_the_oracle(w, h, nx, ny, size, scale):
    sc = scenes.dam_break_2d(nx=nx, ny=ny, box=(0.64, 0.64))
    sim = FluidSim(sc)
    sim.init()
    sim.step(3)
    view = dict(angle=0.1, pos=(0.32, -0.32), scale=scale)
    style = style_for(sc, render_h=size * sc.h)
    rng = np.random.default_rng(w)
    # dark sprites (the blend adds their colour in full) of different colours,
    # thin enough that those below show
    style["colors"][:, :12] = rng.uniform(0.0, 0.15, size=(len(sc.materials), 12))
    style["colors"][:, 3::4] = rng.uniform(0.2, 0.5, size=(len(sc.materials), 3))
    img = sim.render(w, h, view, style)
    ref = oracle_frame(sim, view, style, w, h)
    assert img.tobytes() == ref.tobytes()
    assert w * h == 1 or len(np.unique(img)) > 5  # the one pixel lies between sprites
