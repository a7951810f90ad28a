"""Batches whose scenes call for larger teams than the launch's grid can hold one of
each: a requested shape of several strips per block has at least 128 threads per
strip, so its launch has fewer and larger blocks than were asked for.  The 257 and
125 strips here want teams of 128 and 32 blocks; four strips per block leave one block
per SM.  Results are those of the same scenes stepped alone, bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
DT = 0.005
SIZES = [(8, 8224), (8, 4000)]


def _member(ifl, w, h):
    g = ifl.FluidSolver(w, h, 0.1)
    rng = np.random.default_rng(h)
    u, v = rng.normal(size=(h, w + 1)), rng.normal(size=(h + 1, w))
    u[:, 0] = u[:, w] = 0.0
    v[0, :] = v[h, :] = 0.0
    g.write_field("u", u)
    g.write_field("v", v)
    g.set_pinned_iterations(4)
    return g


@pytest.mark.parametrize("shape", [(128, 4, 2), (256, 8, 2)], ids=lambda s: "%dx%dx%d" % s)
def test_teams_larger_than_the_grid_can_hold(ifl, shape):
    alone = [_member(ifl, w, h) for w, h in SIZES]
    members = [_member(ifl, w, h) for w, h in SIZES]
    b = ifl.Batch(members, threads=shape[0], strips_per_block=shape[1], stages=shape[2])
    b.update(DT)
    for g, m in zip(alone, members):
        g.update(DT)
        assert m.stats()[0] == g.stats()[0]
        for name in ("p", "u", "v"):
            assert np.array_equal(m.read_field(name), g.read_field(name)), (m.w, m.h, name)
