"""The FP64 kick's square roots, quotients and products formed outside the FP64 pipe
(fp64_exact.cuh): the oracle's bits at the block shapes' edges and at the operands that
leave the fast forms' range."""
import numpy as np
import pytest

from oracle import oracle as O
from swiftest_gb300 import SWG_FP64
from swiftest_gb300 import initial_conditions as IC
from swiftest_gb300.api import NBodySystem

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a).view(np.uint64)


def _inputs(kind, n):
    rng = np.random.default_rng(n)
    _, pl, _ = IC.make_system(seed=n, npl=n, ntp=0, mmin=1e-12, mmax=1e-6)
    r, g, R = pl["rh"].copy(), pl["Gmass"].copy(), pl["radius"].copy()
    if kind == "coplanar":  # zero displacements, zero masses
        r[:, 2] = 0.0
        g[::3] = 0.0
    elif kind == "grid":  # round mantissas: powers of two and exact squares
        r = rng.integers(-4, 5, (n, 3)) * 0.5 + np.arange(n)[:, None] * 8.0
        g = 2.0 ** rng.integers(-30, 3, n)
    elif kind == "scales":  # exponents in and out of the fast range, radii from none to large
        r *= 2.0 ** rng.choice([-70, -55, -45, 0, 0, 45, 55, 70], n)[:, None]
        g *= 2.0 ** rng.choice([-120, 0, 60, 110], n)
        R = np.where(rng.random(n) < 0.3, 0.0, R * 2.0 ** rng.choice([-130, 0, 0, 8, 12], n))
    elif kind == "huge":  # squares beyond the doubles' range, exponents that wrap around
        r *= 2.0 ** rng.choice([0, 0, 60, 103, 510, 513, 600], n)[:, None]
        r[::4, 1:] = 0.0
    elif kind == "ties":  # x: zero; y^2: half a unit in the last place of z^2
        r[:] = 0.0
        r[1:, 1] = 2.0 ** -76
        r[1:, 2] = 2.0 ** -49.5 * (1.0 + rng.uniform(0.01, 0.4, n - 1))
        g = rng.uniform(1.0, 2.0, n) * 2.0 ** -90
    elif kind == "close":  # near and overlapping pairs
        r[1::2] = r[: 2 * (n // 2) : 2] * (1.0 + 2.0 ** -rng.integers(8, 45, n // 2))[:, None]
    return r, g, R


@pytest.mark.parametrize("kind", ["disk", "coplanar", "grid", "scales", "close", "huge", "ties"])
@pytest.mark.parametrize("n", [3, 10, 11, 31, 32, 33, 65, 321])
def test_kick_pl_bits(ctx, kind, n):
    r, g, R = _inputs(kind, n)
    for rad in (None, R):
        for nplm in (n, n // 3):  # both loop shapes
            a = ctx.kick_getacch_int_all_tri_pl(r, g, rad, nplm=nplm, precision=SWG_FP64)
            assert np.array_equal(_bits(a), _bits(O.kick_tri_pl(r, g, rad, nplm=nplm)))


@pytest.mark.parametrize("kind", ["disk", "coplanar", "grid", "scales", "huge", "ties"])
@pytest.mark.parametrize("ntp,npl", [(1, 33), (10, 32), (11, 64), (331, 97), (3001, 5)])
def test_kick_tp_bits(ctx, kind, ntp, npl):
    r, g, _ = _inputs(kind, ntp + npl)
    m = (np.arange(ntp) % 4 != 2).astype(np.int32)
    acc = np.random.default_rng(1).normal(size=(ntp, 3)) * 1e-3
    a = ctx.kick_getacch_int_all_tp(r[npl:], r[:npl], g[:npl], lmask=m, acc=acc, precision=SWG_FP64)
    assert np.array_equal(_bits(a), _bits(O.kick_tp(r[npl:], r[:npl], g[:npl], lmask=m, acc=acc)))


@pytest.mark.parametrize("n", [39999, 40001])  # both forms of the drift kernels' dispatch
@pytest.mark.parametrize("dt", [0.003, 0.08])
def test_drift_forms(ctx, n, dt):
    rng = np.random.default_rng(n)
    a, e = rng.uniform(0.4, 5.0, n), rng.uniform(0.0, 0.5, n)
    inc = np.where(np.arange(n) % 5 == 0, 0.0, 0.01)  # zero z components among them
    r, v = IC.el2xv(IC.GMCB, a, e, inc, *rng.uniform(0, 2 * np.pi, (3, n)))
    x, w, f = ctx.drift_all(IC.GMCB, r, v, dt)
    ox, ow, of = O.drift_all(IC.GMCB, r, v, dt)
    assert np.array_equal(f, of)
    small = IC.GMCB / a ** 3 * dt * dt < 0.1  # the branch without CUDA's math functions: same bits
    assert np.array_equal(_bits(x[small]), _bits(ox[small])) and np.array_equal(_bits(w[small]), _bits(ow[small]))
    assert np.abs(x - ox).max() < 1e-9 and np.abs(w - ow).max() < 1e-8
    # the mixed path's form, through a step whose one massive body pulls by 1e-13 of the
    # central body: a few units in the last place over kick and drift
    cb, pl, _ = IC.make_system(seed=1, npl=1, ntp=0, mmin=1e-13, mmax=1.1e-13)
    got = []
    for prec in ("FP64", "MIXED"):
        s = NBodySystem(ctx, "HELIO", cb, pl, {"rh": r, "vh": v}, dt=dt, lclose=False, precision=prec)
        s.step(1)
        got.append(s.get_tp())
        s.close()
    (xr, vr, sr), (xm, vm, sm) = got
    assert np.array_equal(sr, sm)
    scale = np.linalg.norm(xr, axis=1, keepdims=True), np.linalg.norm(vr, axis=1, keepdims=True)
    # 64 units in the last place: a velocity of 2 pi a^-1/2 moves the body by up to 0.4 (3 for
    # the large steps) of its radius, so errors of a few units in mean motion stay below
    assert (np.abs(xm - xr) / scale[0]).max() < 64 * 2.0 ** -52
    assert (np.abs(vm - vr) / scale[1]).max() < 64 * 2.0 ** -52
