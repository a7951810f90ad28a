"""FP32-form PCG (k_pcg32.cu) at the edges of its tiles (2 columns x 4 rows) and
strips (128 rows) against the oracle's FP64 solve.

Bar: the FP32 form's, 1e-4 of the largest pressure difference in the domain
(the closed domain fixes the pressure up to a constant), after as many
iterations as the oracle takes.  The right-hand side is the divergence of
smooth velocities, so that the reference's tolerance of 1e-5 is far above what
FP32 operands lose on these sizes.
"""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_parity import DT, make_gpu, upload

pytestmark = pytest.mark.gpu

# one tile and less, ragged tiles, one strip and less, a strip and a row, more strips than two
SIZES = [(2, 2), (3, 5), (9, 4), (64, 3), (2, 130), (63, 127), (64, 128), (65, 129), (33, 257), (31, 390)]


def _flow(w, h, seed):
    """Closed smooth velocities that are not divergence free."""
    rng = np.random.default_rng(seed)
    a = rng.normal(size=(3, 3))
    x, y = np.arange(w + 1) / w, (np.arange(h) + 0.5) / h
    u = sum(a[i, j] * np.outer(np.cos(np.pi * (j + 1) * y), np.sin(np.pi * (i + 1) * x)) for i in range(3) for j in range(3))
    x, y = (np.arange(w) + 0.5) / w, np.arange(h + 1) / h
    v = sum(a[j, i] * np.outer(np.sin(np.pi * (i + 1) * y), np.cos(np.pi * (j + 1) * x)) for i in range(3) for j in range(3))
    u[:, [0, -1]] = 0.0
    v[[0, -1], :] = 0.0
    return u, v


def _oracle(variant, w, h, bodies):
    o = O.OracleSolver(variant, w, h)
    if bodies:
        o.set_bodies(bodies)
    u, v = _flow(w, h, w * 1000 + h)
    o.array(O.QU, O.A_SRC)[...] = u
    o.array(O.QV, O.A_SRC)[...] = v
    if variant >= 6:
        o.array(O.QT, O.A_SRC)[...] += 40.0 * np.outer(np.sin(np.arange(h) / 5.0), np.cos(np.arange(w) / 7.0))
    return o


def _spread(a, mask):
    return a[mask] - a[mask].mean()


@pytest.mark.parametrize("size", SIZES, ids=lambda s: "%dx%d" % s)
def test_pressure_at_tile_and_strip_edges(ifl, size):
    w, h = size
    o = _oracle(3, w, h, [])
    g = make_gpu(ifl, 3, w, h, [], precision=ifl.FP32)
    upload(ifl, g, o, 3)
    for ph in (O.PH_RHS, O.PH_MATRIX, O.PH_PRECON, O.PH_PROJECT):
        o.phase(ph, DT)
    g.set_pinned_iterations(o.stats()[0][0])
    for ph in (ifl.PH_RHS, ifl.PH_MATRIX, ifl.PH_PRECON, ifl.PH_PROJECT):
        g.run_phase(ph, DT)
    assert g.stats()[2] & 1 == 0
    every = np.ones((h, w), dtype=bool)
    a, b = _spread(g.read_field("p"), every), _spread(o.array(0, O.A_P), every)
    assert np.abs(a - b).max() <= 1e-4 * np.abs(b).max()


@pytest.mark.parametrize("variant,size", [(4, (65, 129)), (6, (131, 67)), (7, (133, 130))], ids=lambda v: str(v))
def test_masked_and_heat_solves(ifl, variant, size):
    """A body in the way (masked coefficients), and from step 6 on the heat solve's
    matrix, whose rows do not sum to zero."""
    w, h = size
    body = [(0, 0.5, 0.5, 0.4, 0.15, 0.6, 0.0, 0.0, 0.0)]
    o = _oracle(variant, w, h, body)
    g = make_gpu(ifl, variant, w, h, body, precision=ifl.FP32)
    upload(ifl, g, o, variant)
    o.update(DT)
    (pi, _, _), (hi, _, _) = o.stats()
    g.set_pinned_iterations(pi, hi)
    g.update(DT)
    assert g.stats()[2] & 1 == 0
    fluid = o.bytes(O.QD, O.B_CELL) == 0
    a, b = _spread(g.read_field("p"), fluid), _spread(o.array(0, O.A_P), fluid)
    assert np.abs(a - b).max() <= 1e-4 * np.abs(b).max()
    if variant >= 6:
        t, s = g.read_field("t"), o.array(O.QT, O.A_SRC)
        assert np.abs(t - s).max() <= 1e-4 * np.abs(s).max()


@pytest.mark.parametrize("shape", [(32, 1, 2), (128, 4, 4), (256, 8, 2)], ids=str)
def test_every_accepted_shape_gives_the_same_bits(ifl, shape):
    """Launch shapes that ask for more strips or stages than a block holds run with
    fewer; the fields do not depend on it."""
    out = []
    for s in (shape, (128, 1, 3)):
        ms = [make_gpu(ifl, 4, w, h, [], precision=ifl.FP32) for w, h in ((70, 300), (133, 64), (40, 520))]
        b = ifl.Batch(ms, threads=s[0], strips_per_block=s[1], stages=s[2], tiles="default")
        for k in range(len(ms)):
            b.set_inflows(k, [(0.3, 0.2, 0.3, 0.05, 1.0, 0.0, 0.0, 2.0)])
        b.update(0.0025)
        assert all(st[2] & 1 == 0 for st in b.stats())
        out.append([m.read_field(n) for m in ms for n in ("u", "v", "p")])
    for a, c in zip(*out):
        assert np.array_equal(a, c)
