"""Step 8's particle-to-grid transfer with hundreds of particles around one node (as
velocities without bound leave them): buckets about the size up to which a thread
sorts its own (256), and far above it, bit for bit the oracle's sums.
"""
import numpy as np
import pytest

import flip_cases as FC
from oracle import oracle as O
from test_gpu_flip import _fields_equal, _pair, _particles_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("crowd", [250, 260, 3000])
@pytest.mark.parametrize("place", ["cell", "corners"])
def test_crowded_nodes(ifl, crowd, place):
    w, h = 32, 24
    o, g, _ = _pair(ifl, w, h, [])
    o.flip_init()
    g.flip_init()
    rng = np.random.default_rng(crowd)
    x, y = o.particles(O.P_X).copy(), o.particles(O.P_Y).copy()
    if place == "cell":  # one base node for each kind of node
        cx, cy = 10.5 + 0.5 * rng.random(crowd), 7.5 + 0.5 * rng.random(crowd)
    else:                # where the advection's clamp leaves what went beyond the domain
        cx = rng.choice([0.0, w - 0.001], crowd)
        cy = rng.choice([0.0, h - 0.001], crowd)
    x, y = np.concatenate([x, cx]), np.concatenate([y, cy])
    perm = rng.permutation(len(x))
    n = len(x)
    arrays = (x[perm], y[perm], rng.random(n), 294.0 + rng.random(n), rng.normal(size=n), rng.normal(size=n))
    o.set_particles(arrays)
    g.set_particles(arrays)
    g.rng_state = o.rng_state
    for ph in (O.PH_FILL_SOLID, O.PH_P2G):
        o.phase(ph, FC.DT)
        g.run_phase(ph, FC.DT)
    _fields_equal(ifl, g, o, "p2g")
    _particles_equal(ifl, g, o, "p2g")
