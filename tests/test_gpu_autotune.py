"""The tuner gives every launch shape it considers the same trials."""
import numpy as np
import pytest

from arphys import FluidSim, scenes

pytestmark = pytest.mark.gpu


def _launches(n):
    sc = scenes.dam_break_2d(nx=n, ny=n, box=(round(0.01 * (2 * n + 2), 6), round(0.01 * (n + 20), 6)))
    sim = FluidSim(sc)
    sim.init()
    before = sim.launch_count()
    sim.autotune()
    return sim.launch_count() - before


def test_every_shape_is_timed_as_often_as_any_other():
    group, both, block = _launches(100), _launches(200), _launches(380)  # 10,000, 40,000 and 144,400 particles
    # 3 shapes of the group form and 12 of the block form, besides the same few launches that order the state
    per_shape, order = divmod(both - group, 12)
    assert order == 0
    rest = group - 3 * per_shape
    assert 0 < rest < 3 * per_shape
    assert both == rest + 15 * per_shape
    assert (block - rest) % 12 == 0
