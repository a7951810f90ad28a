"""FP64-form PCG (k_pcg64.cu) at the edges of its strips (32 rows) and ring blocks (8
diagonals): the plain step, whose solve has the L D L^T form, against the oracle
after as many iterations.  Bar: 1e-10 of the largest pressure difference, the one
that the iteration-cap test holds this form to on plain systems.
"""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_parity import DT, make_gpu, upload
from test_gpu_pcg32 import _oracle, _spread

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(2, 2), (9, 31), (8, 32), (33, 33), (40, 64), (17, 65), (120, 97), (31, 290)],
                         ids=lambda s: "%dx%d" % s)
def test_pressure_at_strip_edges(ifl, size):
    w, h = size
    o = _oracle(3, w, h, [])
    g = make_gpu(ifl, 3, w, h, [])
    upload(ifl, g, o, 3)
    for ph in (O.PH_RHS, O.PH_MATRIX, O.PH_PRECON, O.PH_PROJECT):
        o.phase(ph, DT)
    g.set_pinned_iterations(o.stats()[0][0])
    for ph in (ifl.PH_RHS, ifl.PH_MATRIX, ifl.PH_PRECON, ifl.PH_PROJECT):
        g.run_phase(ph, DT)
    assert g.stats()[2] & 1 == 0
    every = np.ones((h, w), dtype=bool)
    a, b = _spread(g.read_field("p"), every), _spread(o.array(0, O.A_P), every)
    assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max()
