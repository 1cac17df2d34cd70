"""The FP64 kick's square roots, quotients and products formed outside the FP64 pipe
(fp64_exact.cuh): the oracle's bits at the block shapes' edges and at the operands that
leave the fast forms' range."""
import numpy as np
import pytest

from oracle import oracle as O
from swiftest_gb300 import SWG_FP64
from swiftest_gb300 import initial_conditions as IC

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
    elif kind == "close":  # near and overlapping pairs
        r[1::2] = r[: 2 * (n // 2) : 2] * (1.0 + 2.0 ** -rng.integers(8, 45, n // 2))[:, None]
    return r, g, R


@pytest.mark.parametrize("kind", ["disk", "coplanar", "grid", "scales", "close"])
@pytest.mark.parametrize("n", [3, 10, 11, 31, 32, 33, 65, 321])
def test_kick_pl_bits(ctx, kind, n):
    r, g, R = _inputs(kind, n)
    for rad in (None, R):
        for nplm in (n, n // 3):  # both loop shapes
            a = ctx.kick_getacch_int_all_tri_pl(r, g, rad, nplm=nplm, precision=SWG_FP64)
            assert np.array_equal(_bits(a), _bits(O.kick_tri_pl(r, g, rad, nplm=nplm)))


@pytest.mark.parametrize("kind", ["disk", "coplanar", "grid", "scales"])
@pytest.mark.parametrize("ntp,npl", [(1, 33), (10, 32), (11, 64), (331, 97), (3001, 5)])
def test_kick_tp_bits(ctx, kind, ntp, npl):
    r, g, _ = _inputs(kind, ntp + npl)
    m = (np.arange(ntp) % 4 != 2).astype(np.int32)
    acc = np.random.default_rng(1).normal(size=(ntp, 3)) * 1e-3
    a = ctx.kick_getacch_int_all_tp(r[npl:], r[:npl], g[:npl], lmask=m, acc=acc, precision=SWG_FP64)
    assert np.array_equal(_bits(a), _bits(O.kick_tp(r[npl:], r[:npl], g[:npl], lmask=m, acc=acc)))
