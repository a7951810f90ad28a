"""The serving loop keeps the first batch's autotuned shape although requests of
that batch finish with its first step (needs a GB300)."""
import pytest

pytestmark = pytest.mark.gpu


def test_shape_is_kept_when_requests_leave_with_the_first_step(ifl):
    srv = ifl.Server(precision=ifl.FP32)
    inflow = [(0.45, 0.2, 0.15, 0.05, 1.0, 0.0, 0.0, 3.0)]
    for steps in (1, 2, 1):
        srv.submit(64, 48, steps, inflows=inflow)
    assert srv.step() == (1, 0)
    info = srv.info()
    assert info["threads"] > 0 and info["stages"] > 0
    assert srv.step() == (0, 0)
    assert {k: srv.info()[k] for k in ("threads", "strips_per_block", "stages")} == \
        {k: info[k] for k in ("threads", "strips_per_block", "stages")}
    assert len(srv.completions()) == 3
