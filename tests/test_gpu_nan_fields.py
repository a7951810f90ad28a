"""NaN velocities and the advection's sample positions: a NaN position (where the
reference converts it to an integer, which C leaves undefined) reads inside the
array and gives a NaN, cells that do not see one keep their values bit for bit, and a
whole update of a scene that has gone NaN comes back without an error.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DT = 0.005
W, H = 40, 33
BODY = (0.55, 0.5, 0.2, 0.15, 0.3, 0.0, 0.0, 0.0)


def _solver(ifl, variant, precision):
    bodies = [ifl.SolidBox(*BODY)] if variant >= 4 else []
    kw = dict(variant=variant, precision=precision)
    if variant >= 7:
        return ifl.FluidSolver(W, H, 0.1, 0.25, 0.01, bodies, **kw)
    return ifl.FluidSolver(W, H, 0.1, bodies, **kw) if bodies else ifl.FluidSolver(W, H, 0.1, **kw)


def _fields(g, nan):
    rng = np.random.default_rng(11)
    f = {"d": rng.random((H, W)), "u": 0.3 * rng.normal(size=(H, W + 1)), "v": 0.3 * rng.normal(size=(H + 1, W))}
    if nan:
        f["u"][5, 6] = np.nan
    for name, a in f.items():
        g.write_field(name, a)


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32"])
@pytest.mark.parametrize("variant", [1, 2, 3, 4, 7])
def test_nan_velocity(ifl, variant, precision):
    out = []
    for nan in (False, True):
        g = _solver(ifl, variant, precision)
        _fields(g, nan)
        if variant >= 4:
            g.run_phase(ifl.PH_FILL_SOLID, DT)
        g.run_phase(ifl.PH_ADVECT, DT)
        out.append({n: g.read_field(n) for n in ("d", "u", "v")})
        if nan:
            g.update(DT)
            g.update(DT)
            assert g.stats()[2] & 1 == 0
    for name in ("d", "u", "v"):
        a, b = out[0][name], out[1][name]
        bad = np.isnan(b)
        assert np.isfinite(a).all()
        # the cells whose backtrace reads the face, a few rows and columns around it
        assert bad.any() and bad[:12, :13].sum() == bad.sum()
        assert np.array_equal(a[~bad], b[~bad])


@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "fp32-solves"])
def test_flip_scene_that_goes_nan(ifl, precision):
    g = ifl.FluidSolver(W, H, 0.1, 0.25, 0.01, [ifl.SolidBox(*BODY)], variant=ifl.FLIP, precision=precision)
    g.flip_init()
    a = [g.particles(k).copy() for k in range(6)]
    a[4][7] = np.nan  # one particle's velocity: the pressure solve spreads it
    g.set_particles(a)
    for _ in range(3):
        g.update(DT)
    assert g.stats()[2] & 1 == 0
    assert np.isnan(g.particles(0)).any() and g.particle_count() <= 12 * W * H


def test_particle_at_a_nan_position(ifl):
    """Grid to particles and the advection: that particle's values and position become NaN, no other's."""
    out = []
    for nan in (False, True):
        g = ifl.FluidSolver(W, H, 0.1, 0.25, 0.01, [ifl.SolidBox(*BODY)], variant=ifl.FLIP)
        g.flip_init()
        a = [g.particles(k).copy() for k in range(6)]
        if nan:
            a[0][9] = np.nan
        g.set_particles(a)
        _fields(g, False)
        for ph in (ifl.PH_FLIP_COPY, ifl.PH_G2P, ifl.PH_PADVECT):
            g.run_phase(ph, DT)
        out.append([g.particles(k) for k in range(6)])
    for a, b in zip(*out):
        assert np.isnan(b[9]) and np.array_equal(np.delete(a, 9), np.delete(b, 9))
