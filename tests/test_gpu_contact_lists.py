"""Contact and friction where a particle's hits are taken in several lists: the
hits with a contact potential are marked list by list and walked a second time."""
import numpy as np
import pytest

from arphys import FluidSim
from arphys.abi import CONTACT_LINEAR
from helpers import rel_err
from oracle.oracle import Oracle
from test_gpu_fluid_forms import block

pytestmark = pytest.mark.gpu


# up to 31, 153 and 162 hits a particle (lists hold 40 to 96), at most 128 particles a cell, which
# is what the oracle's buckets hold; contacts of one material pair, then of every pair, the particle's
# own material among them
@pytest.mark.parametrize("n,cells", [(300, 2), (1800, 2), (6000, 3)])
@pytest.mark.parametrize("every_pair", [False, True])
def test_contacts_of_full_lists_match_the_oracle_in_every_form(n, cells, every_pair):
    sc = block(n, 3, cells, seed=n, wall=True)
    if every_pair:
        for i in (1, 2):
            sc.interactions[i, i] = (CONTACT_LINEAR, 700.0, 0.03, 0.1, 0.0)
            sc.interaction_given[i, i] = 1
    ref = None
    for v in range(FluidSim.fluid_variant_count()):
        sim = FluidSim(sc)
        sim.init()
        sim.set_fluid_variant(v)
        sim.step(2)
        p = sim.particles()
        ref = p if ref is None else ref
        assert p.tobytes() == ref.tobytes(), v
    r, r32 = [], []
    for bits, out in ((64, r), (32, r32)):
        o = Oracle(sc, bits)
        o.step(2)
        out.append(o.state())
    for key in ("den", "pos", "vel"):
        # as close to the double oracle as twice the float oracle is, or 1e-6
        assert rel_err(ref[key], r[0][key]) <= max(1e-6, 2.0 * rel_err(r32[0][key], r[0][key])), key
