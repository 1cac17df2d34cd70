"""TRIANGULAR checks of one pair of lists on both sides of the line from which they go over
radius-sorted tiles (encounter.cu SORTED_PAIRS): the oracle's lists, with segments, sub-tiles
and receiver tiles left partly filled, and with bodies whose bounds are not finite."""
import numpy as np
import pytest

from oracle import oracle as O
from swiftest_gb300 import initial_conditions as IC

pytestmark = pytest.mark.gpu


def _disk(seed, npl, ntp):
    _, pl, tp = IC.make_system(seed=seed, npl=npl, ntp=ntp, amin=0.3, amax=3.0)
    return pl["rh"], pl["vh"], 3.0 * pl["rhill"], tp["rh"], tp["vh"]


def _odd(r, v, renc=None):
    """NaN and infinite positions and velocities, coincident and distant bodies, odd radii."""
    n = len(r)
    r[5], v[7] = np.nan, np.nan
    r[8, 1], v[9, 2] = np.inf, -np.inf
    r[11] = r[7] * (1 + 1e-9)  # within the radius of the body without a velocity
    r[13] = r[9] * (1 - 1e-9)
    r[n // 2] = r[n - 1]
    r[n // 3] *= 1e25
    if renc is not None:
        renc[3], renc[4], renc[20], renc[21] = 0.0, np.nan, 0.6, -0.3


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("n", [6300, 6337, 8193])  # below and above the line, past a segment
def test_plpl(ctx, n, odd):
    r, v, renc, _, _ = _disk(n, n, 0)
    if odd:
        _odd(r, v, renc)
    g = ctx.encounter_check_all_plpl(r, v, renc, 0.005)
    o = O.encounter_plpl(r, v, renc, 0.005)
    assert len(o[0]) > 1024  # the first raw buffer overflows
    for a, b in zip(g, o):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("npl,ntp", [(499, 40001), (501, 40001), (33, 700001), (20011, 1025)])
def test_pltp(ctx, npl, ntp, odd):
    r, v, renc, tr, tv = _disk(npl, npl, ntp)
    if odd and npl > 33:
        _odd(r, v, renc)
        _odd(tr, tv)
        tr[31], tr[32] = r[7] * (1 + 1e-9), r[9] * (1 + 1e-9)
    g = ctx.encounter_check_all_pltp(r, v, tr, tv, renc, 0.005, cap=200000)
    o = O.encounter_pltp(r, v, tr, tv, renc, 0.005)
    assert len(o[0]) > 0
    for a, b in zip(g, o):
        assert np.array_equal(a, b)
