"""HELIO steps of one system taken in one call, where a step's discard scan runs beside the
massive bodies' next step, and WHM steps, whose test particles run beside the massive bodies: the
same bits as steps taken one call each and as steps on one
stream (the profiled form), discards among them."""
import numpy as np
import pytest

from swiftest_gb300 import initial_conditions as IC
from swiftest_gb300.api import NBodySystem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("integrator", ["HELIO", "WHM"])
@pytest.mark.parametrize("precision", ["FP64", "MIXED"])
@pytest.mark.parametrize("npl,ntp", [(1, 1), (33, 65), (100, 1000)])
def test_same_bits(ctx, npl, ntp, precision, integrator):
    cb, pl, tp = IC.make_system(seed=npl, npl=npl, ntp=ntp, amin=0.8, amax=1.2, mmin=1e-9, mmax=1e-6)
    pl = IC.sort_for_integrator(pl, integrator)
    pl["radius"] = pl["radius"] * 1000.0  # test particles hit massive bodies
    got = []
    for form in ("row", "single", "one stream"):
        s = NBodySystem(ctx, integrator, cb, pl, tp, dt=0.005, lclose=True, precision=precision)
        if form == "one stream":
            s.profile(True)
        for n in (40,) if form != "single" else (1,) * 40:
            s.step(n)
        got.append((*s.get_pl(), *s.get_tp()))
        assert ntp < 1000 or s.stats()["collisions"] > 0
        s.close()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))
