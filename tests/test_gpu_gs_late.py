"""The Gauss-Seidel solve (k_gs.cu) where it converges late: with many sweeps in flight,
some workers have begun their last sweep when the verdict comes and others have
not, and the sweeps that the cap would allow never run.  Sweep count, last
maximum change and pressure are the oracle's, bit for bit.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
DT = 0.005
# one strip, two, five (the last of two rows), and a row-heavy one
SIZES = [(40, 20), (64, 64), (33, 130), (200, 64)]
# sweeps from far before the cap of 600 to the cap: the ones in flight are 32 to 116, their lead
# over the verdict is 43 to 141, so both ends of what may still run at the cap lie in between
COUNTS = [2, 250, 345, 400, 441, 459, 470, 481, 490, 505, 523, 527, 540, 557, 580, 598, 599, 600]


def _oracle(w, h, scale):
    rng = np.random.default_rng(w * 1000 + h)
    u, v = rng.normal(size=(h, w + 1)), rng.normal(size=(h + 1, w))
    u[:, 0] = u[:, w] = 0.0  # closed walls: the system is consistent
    v[0, :] = v[h, :] = 0.0
    o = O.OracleSolver(2, w, h)
    o.array(O.QU, O.A_SRC)[...] = u * scale
    o.array(O.QV, O.A_SRC)[...] = v * scale
    o.phase(O.PH_RHS, DT)
    o.phase(O.PH_PROJECT, DT)
    return o


def _scaled_to(w, h, sweeps):
    """The oracle's solve for the scale of the velocities at which it takes `sweeps` sweeps."""
    lo, hi = 1e-8, 1e3
    for _ in range(80):
        mid = (lo * hi) ** 0.5
        o = _oracle(w, h, mid)
        it, st, _ = o.stats()[0]
        if it == sweeps and st == O.PCG_CONVERGED:
            return mid, o
        lo, hi = (mid, hi) if it < sweeps else (lo, mid)
    raise AssertionError("no scale takes %d sweeps" % sweeps)


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "%dx%d" % s)
def test_converges_late(ifl, size):
    w, h = size
    for sweeps in COUNTS:
        scale, o = _scaled_to(w, h, sweeps)
        rng = np.random.default_rng(w * 1000 + h)
        u, v = rng.normal(size=(h, w + 1)), rng.normal(size=(h + 1, w))
        u[:, 0] = u[:, w] = 0.0
        v[0, :] = v[h, :] = 0.0
        g = ifl.FluidSolver(w, h, 0.1, variant=ifl.GS)
        g.set_wait_limit(1 << 20)
        g.write_field("u", u * scale)
        g.write_field("v", v * scale)
        g.run_phase(ifl.PH_RHS, DT)
        g.run_phase(ifl.PH_PROJECT, DT)
        assert g.stats()[0] == o.stats()[0], sweeps
        assert g.stats()[2] == 0
        assert np.array_equal(g.read_field("p"), o.array(0, O.A_P)), sweeps
        g.close()
