"""The order-exact extrapolation of step 8 (k_fields.cu, extrap_lifo_kernel) in each of
its forms: values after the walk (small grids), value by value with the cells' bytes
in shared memory (larger ones, and small ones with more than 4096 pops), and in
global memory (more than 160 KB of bytes).  Bit for bit the oracle's, from the
crafted particle state with empty cells.
"""
import pytest

import flip_cases as FC
from oracle import oracle as O
from test_gpu_flip import _fields_equal, _pair, _particles_equal, _random_fields

pytestmark = pytest.mark.gpu
BLOCK = (0, 0.5, 0.5, 0.7, 0.7, 0.3, 0.0, 0.0, 0.0)


@pytest.mark.parametrize("w,h,body", [(64, 50, FC.BOX), (128, 128, FC.BOX), (160, 150, BLOCK), (400, 390, FC.BOX),
                                      (410, 405, FC.BOX)])
def test_transfer_with_empty_cells(ifl, w, h, body):
    o, g, _ = _pair(ifl, w, h, [body])
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
