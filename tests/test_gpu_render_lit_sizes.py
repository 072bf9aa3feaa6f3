"""Lit frames with sprites around the size from which several threads share one, and
larger than the frame, against the oracle."""
import numpy as np
import pytest

from arphys import FluidSim, scenes
from test_gpu_render import oracle_frame, style_for

pytestmark = pytest.mark.gpu


# sprite sizes in pixels of min(w, h); 16.0 = 0.125 * 128 exactly
@pytest.mark.parametrize("w,h,size", [(128, 150, 2.5), (128, 150, 16.0), (128, 150, 16.01), (97, 128, 30.3),
                                      (128, 97, 75.0), (64, 90, 400.0)])
def test_lit_frames_of_every_sprite_size_match_the_oracle(w, h, size):
    sc = scenes.small_fluid_bar_3d()
    sim = FluidSim(sc)
    sim.init()
    sim.step(2)
    b, d = sc.bounds_min[:3], sc.bounds_dim[:3]
    view = dict(angle=0.3, pos=(b[0] + 0.5 * d[0], -(b[1] + 0.5 * d[1])), scale=1.2)
    style = style_for(sc, lighting=True, render_h=size / min(w, h))
    img = sim.render(w, h, view, style).astype(int)
    ref = oracle_frame(sim, view, style, w, h).astype(int)
    assert (ref != 255).any()
    assert np.abs(img - ref).max() <= 1  # the shading's contracted multiply-adds: one 8-bit level
