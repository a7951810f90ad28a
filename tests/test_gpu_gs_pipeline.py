"""The Gauss-Seidel solve's sweeps in flight (k_gs.cu) at the edges of its strips (32
rows) and of its pipeline, and beyond the range of its fast division: the sweep
count, the last maximum change and every value are the oracle's, bit for bit (the
solve does the reference's operations in the reference's order).
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
DT = 0.005

# less than a strip, a strip and a row, more strips than columns, more columns than rows
SIZES = [(2, 2), (3, 32), (31, 33), (32, 64), (33, 65), (5, 200), (200, 5), (97, 31)]


def _pair(ifl, w, h, scale=1.0):
    rng = np.random.default_rng(w * 1000 + h)
    u, v = rng.normal(size=(h, w + 1)) * scale, rng.normal(size=(h + 1, w)) * scale
    p = rng.normal(size=(h, w)) * scale
    o, g = O.OracleSolver(2, w, h), ifl.FluidSolver(w, h, 0.1, variant=ifl.GS)
    o.array(O.QU, O.A_SRC)[...] = u
    o.array(O.QV, O.A_SRC)[...] = v
    o.array(0, O.A_P)[...] = p
    g.write_field("u", u)
    g.write_field("v", v)
    g.write_field("p", p)
    return o, g


def _solve(ifl, o, g):
    for ph_o, ph_g in ((O.PH_RHS, ifl.PH_RHS), (O.PH_PROJECT, ifl.PH_PROJECT)):
        o.phase(ph_o, DT)
        g.run_phase(ph_g, DT)
    assert g.stats()[0] == o.stats()[0]
    assert g.stats()[2] == 0
    assert np.array_equal(g.read_field("p"), o.array(0, O.A_P))


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "%dx%d" % s)
def test_edges_of_strips_and_pipeline(ifl, size):
    o, g = _pair(ifl, *size)
    _solve(ifl, o, g)  # from p as written
    _solve(ifl, o, g)  # from the solution: the first sweeps decide


def _sweeps(p, r, scale, n):
    """The reference's loop (1-matrixless/Fluid.cpp:192-240), n times, in Python's doubles."""
    p = p.copy()
    h, w = p.shape
    for _ in range(n):
        for y in range(h):
            for x in range(w):
                diag, off = 0.0, 0.0
                for ok, yy, xx in ((x > 0, y, x - 1), (y > 0, y - 1, x), (x < w - 1, y, x + 1), (y < h - 1, y + 1, x)):
                    if ok:
                        diag += scale
                        off -= scale * p[yy, xx]
                p[y, x] = (r[y, x] - off) / diag
    return p


@pytest.mark.parametrize("sweeps", [0, 1, 2, 7, 30])
def test_pinned_counts(ifl, sweeps):
    w, h = 9, 35
    _, g = _pair(ifl, w, h)
    g.set_pinned_iterations(sweeps, -1)
    g.run_phase(ifl.PH_RHS, DT)
    want = _sweeps(g.read_field("p"), g.read_field("r"), DT / (0.1 * (1.0 / min(w, h)) ** 2), sweeps)
    g.run_phase(ifl.PH_PROJECT, DT)
    assert g.stats()[0][0] == sweeps
    assert np.array_equal(g.read_field("p"), want)


@pytest.mark.parametrize("scale", [1e-300, 1e-310, 1e200, 1e300])
def test_operands_outside_the_fast_division(ifl, scale):
    o, g = _pair(ifl, 40, 35, scale)
    for ph_o, ph_g in ((O.PH_RHS, ifl.PH_RHS), (O.PH_PROJECT, ifl.PH_PROJECT)):
        o.phase(ph_o, DT)
        g.run_phase(ph_g, DT)
    assert g.stats()[0][0] == o.stats()[0][0]
    a, b = g.read_field("p"), o.array(0, O.A_P)
    assert np.array_equal(a, b, equal_nan=True)
