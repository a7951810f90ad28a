"""The order-exact extrapolation of step 8 (k_fields.cu, extrap_walk) in both places
that its bytes can lie: shared memory, and global memory for grids above 160 KB of
them.  Bit for bit the oracle's, from the crafted particle state with empty cells.  (Sizes
with h <= w + 2: step 7-8 index v-face densities with the u width.)
"""
import pytest

import flip_cases as FC
from oracle import oracle as O
from test_gpu_flip import _fields_equal, _pair, _particles_equal, _random_fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(64, 50), (128, 128), (400, 390), (410, 405)], ids=lambda s: "%dx%d" % s)
def test_transfer_with_empty_cells(ifl, size):
    w, h = size
    o, g, _ = _pair(ifl, w, h, [FC.BOX])
    o.flip_init()
    g.flip_init()
    arrays = FC.crafted(w, h, o.particles(O.P_X).copy(), o.particles(O.P_Y).copy())
    o.set_particles(arrays)
    g.set_particles(arrays)
    _random_fields(ifl, g, o, 1)
    for ph in (O.PH_FILL_SOLID, O.PH_P2G):
        o.phase(ph, FC.DT)
        g.run_phase(ph, FC.DT)
    _fields_equal(ifl, g, o, "p2g")
    _particles_equal(ifl, g, o, "p2g")
    assert g.stats()[2] & 0xC == 0
