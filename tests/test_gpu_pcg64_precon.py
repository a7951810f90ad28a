"""The FP64 form's factor and one application of its preconditioner in scenes with
bodies (steps 4-7), whose solves keep the reference's own arithmetic (k_pcg64.cu): bit
for bit the oracle's on the fluid cells, at the edges of strips (32 rows) and ring
blocks (8 diagonals), where the boundary rows pass from strip to strip.  A solve that
is pinned to no iteration ends after z = M^-1 r.
"""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_parity import DT, make_gpu, upload
from test_gpu_pcg32 import _oracle

pytestmark = pytest.mark.gpu
BODY = [(0, 0.5, 0.5, 0.4, 0.15, 0.6, 0.0, 0.0, 0.0)]


@pytest.mark.parametrize("size", [(33, 31), (33, 32), (24, 33), (64, 65), (61, 64), (40, 97), (130, 128), (17, 290)],
                         ids=lambda s: "%dx%d" % s)
@pytest.mark.parametrize("variant", [4, 5, 6, 7])
def test_preconditioner_in_reference_arithmetic(ifl, variant, size):
    w, h = size
    if variant == 7:  # step 7's index of the v-face densities needs h < w + 2
        w, h = max(w, h), min(w, h)
    o = _oracle(variant, w, h, BODY)
    g = make_gpu(ifl, variant, w, h, BODY)
    for ph in (O.PH_FILL_SOLID, O.PH_BC, O.PH_RHS, O.PH_DENSITIES, O.PH_MATRIX):
        if ph != O.PH_DENSITIES or variant == 7:
            o.phase(ph, DT)
    upload(ifl, g, o, variant)
    g.run_phase(ifl.PH_MATRIX, DT)  # the neighbour bits
    o.set_pinned_iterations(0, 0)
    g.set_pinned_iterations(0, 0)
    for ph_o, ph_g in ((O.PH_PRECON, ifl.PH_PRECON), (O.PH_PROJECT, ifl.PH_PROJECT)):
        o.phase(ph_o, DT)
        g.run_phase(ph_g, DT)
    assert g.stats()[2] & 1 == 0
    fluid = o.bytes(O.QD, O.B_CELL) == 0
    assert 0 < fluid.sum() < w * h
    assert np.array_equal(g.read_field("precon")[fluid], o.array(0, O.A_PRECON)[fluid])
    z = g.read_field(ifl.F_Z)
    assert np.abs(z[fluid]).max() > 0
    assert np.array_equal(z[fluid], o.array(0, O.A_Z)[fluid])
