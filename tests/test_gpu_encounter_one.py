"""SORTSWEEP checks at the edges of the merge sort's tiles and rounds and of its range, and
TRIANGULAR checks of one pair of lists on both sides of the line from which they go over
radius-sorted tiles (encounter.cu SORTED_PAIRS): the oracle's lists, with segments, sub-tiles
and receiver tiles left partly filled, and with bodies whose bounds are not finite."""
import numpy as np
import pytest

from oracle import oracle as O
from swiftest_gb300 import SWG_ENC_SORTSWEEP, SWG_ENC_TRIANGULAR
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
@pytest.mark.parametrize("n", [4470, 4473, 6300, 6337, 8193])  # below and above the line, past a segment
def test_plpl(ctx, n, odd):
    r, v, renc, _, _ = _disk(n, n, 0)
    if odd:
        _odd(r, v, renc)
    g = ctx.encounter_check_all_plpl(r, v, renc, 0.005)
    o = O.encounter_plpl(r, v, renc, 0.005)
    assert n < 6300 or len(o[0]) > 1024  # the first raw buffer overflows
    for a, b in zip(g, o):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("npl,ntp", [(249, 40001), (251, 40001), (499, 40001), (501, 40001), (33, 700001), (20011, 1025)])
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


# extents (two per body): one tile of 512 and its edge, one, two, three and four merge rounds, past
# the range (the radix sort)
@pytest.mark.parametrize("npl,ntp", [(1, 1), (7, 248), (7, 249), (7, 250), (50, 1998), (50, 1999), (33, 16351),
                                     (33, 16352), (31, 131041), (31, 131042), (20, 262124), (20, 262125)])
def test_pltp_sortsweep(ctx, npl, ntp):
    r, v, renc, tr, tv = _disk(npl + ntp, npl, ntp)
    tr[::1 + ntp // 200] = tr[0]  # equal extents in many tiles
    if npl > 6:
        r[3] = r[5]
        tr[1::2 + ntp // 100] = r[5] * (1 + 1e-4)
    g = ctx.encounter_check_all_pltp(r, v, tr, tv, renc, 0.005, mode=SWG_ENC_SORTSWEEP, cap=200000)
    o = O.encounter_pltp(r, v, tr, tv, renc, 0.005, mode=SWG_ENC_SORTSWEEP)
    assert npl == 1 or len(o[0]) > 0
    for a, b in zip(g, o):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("n", [2, 255, 256, 257, 2049, 16385])
def test_plpl_sortsweep(ctx, n):
    r, v, renc, _, _ = _disk(n, n, 0)
    few = slice(0, n, 1 + n // 50)
    r[few], renc[few] = r[0], renc[0]  # coincident bodies
    r[1 : n : 1 + n // 20] *= 0.0  # extents around zero
    g = ctx.encounter_check_all_plpl(r, v, 0.1 * renc, 0.005, mode=SWG_ENC_SORTSWEEP, cap=10000)
    o = O.encounter_plpl(r, v, 0.1 * renc, 0.005, mode=SWG_ENC_SORTSWEEP)
    for a, b in zip(g, o):
        assert np.array_equal(a, b)


# lists of one block's sort and its edge, one and two merge rounds and their edge, with every pair
# found from both sides by the sweep
@pytest.mark.parametrize("mode", [SWG_ENC_TRIANGULAR, SWG_ENC_SORTSWEEP])
@pytest.mark.parametrize("m,n", [(1, 1), (2, 1), (32, 64), (7, 293), (45, 91), (64, 65), (90, 400)])
def test_list_lengths(ctx, m, n, mode):
    rng = np.random.default_rng(m * n)
    r, tr = rng.normal(size=(m, 3)) * 1e-3 + [1.0, 0, 0], rng.normal(size=(n, 3)) * 1e-3 + [1.0, 0, 0]
    v, tv = rng.normal(size=(m, 3)), rng.normal(size=(n, 3))
    renc = np.full(m, 0.5)  # every pair
    g = ctx.encounter_check_all_pltp(r, v, tr, tv, renc, 0.005, mode=mode, cap=40000)
    o = O.encounter_pltp(r, v, tr, tv, renc, 0.005, mode=mode)
    assert len(o[0]) == m * n or mode == SWG_ENC_SORTSWEEP
    for a, b in zip(g, o):
        assert np.array_equal(a, b)
