"""The allocation-free solve on matrices whose entries beyond the grid are not zero.

A caller may fill aPlusX and aPlusY with one value everywhere: buildPreconditioner
reads the entries of the last column and row (3-conjugate-gradients/Fluid.cpp:253-264),
the substitutions and the matvec guard them by x < w - 1 and y < h - 1 (:284-303,
:315-332).  Sizes: a last strip (32 rows) that is full, whose top lane has no
neighbour to take from, and one that is not.  Bars: those of test_zz_no_alloc.py, the
oracle's iteration count and 1e-10 of the largest pressure.
"""
import numpy as np
import pytest

from oracle import oracle as O
from test_zz_no_alloc import DT, TOL, _noalloc, _velocities

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(24, 32), (32, 32), (33, 64), (24, 40), (2, 32), (130, 96)], ids=lambda s: "%dx%d" % s)
def test_entries_of_neighbours_that_do_not_exist(ifl, size):
    torch = pytest.importorskip("torch")
    w, h = size
    o = O.OracleSolver(O.PLAIN, w, h)
    u, v = _velocities(w, h, 1)
    o.array(O.QU, O.A_SRC)[...] = u
    o.array(O.QV, O.A_SRC)[...] = v
    o.phase(O.PH_RHS, DT)
    o.phase(O.PH_MATRIX, DT)
    ax, ay = o.array(0, O.A_APLUSX), o.array(0, O.A_APLUSY)
    ax[:, w - 1] = ay[h - 1, :] = ay[0, 0]
    arrays = [o.array(0, k).copy() for k in (O.A_ADIAG, O.A_APLUSX, O.A_APLUSY, O.A_R)]
    o.phase(O.PH_PRECON, DT)
    o.phase(O.PH_PROJECT, DT)
    it_o, st_o, _ = o.stats()[0]
    rc, got, it, st = _noalloc(ifl, torch, w, h, arrays)
    assert rc == ifl.OK
    assert (it, st) == (it_o, st_o)
    p = o.array(0, O.A_P)
    assert np.abs(got - p).max() <= TOL * np.abs(p).max()
