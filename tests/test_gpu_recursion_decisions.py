"""The recursion's list and collision checks decide most pairs in FP32 (symba_dev.cuh
d_list_pair, d_collision_far): at thresholds the decisions, and so the FP64 path's bits, are
the oracle's."""
import numpy as np
import pytest

from oracle import oracle as O
from swiftest_gb300 import initial_conditions as IC
from swiftest_gb300.api import NBodySystem

pytestmark = pytest.mark.gpu


def _pairs(kind, n=12):
    """n pairs of bodies on circular orbits well apart, each pair's second body displaced by a
    multiple of the mutual Hill radius (grazing the encounter radius and the shells below it, to
    1e-6 and to a few ulps), at rest, approaching, receding or almost tangential."""
    rng = np.random.default_rng({"still": 1, "approach": 2, "recede": 3, "tangent": 4}[kind])
    a = 0.4 + 0.25 * np.arange(n)
    m = 10.0 ** rng.uniform(-9, -7, (n, 2))
    th = rng.uniform(0, 2 * np.pi, n)
    r, v, gm = [], [], []
    for k in range(n):
        mu = IC.GMCB
        x = a[k] * np.array([np.cos(th[k]), np.sin(th[k]), 0.0])
        w = np.sqrt(mu / a[k]) * np.array([-np.sin(th[k]), np.cos(th[k]), 0.0])
        rh = a[k] * ((m[k] / 3.0) ** (1 / 3)).sum()
        d = rng.normal(size=3)
        d /= np.linalg.norm(d)
        e = np.cross(d, rng.normal(size=3))
        e /= np.linalg.norm(e)
        sep = rh * 0.48075 ** (k % 4) * (1.0 + [0.0, 1e-6, -1e-6, 3e-16][k % 4])
        speed = rng.uniform(0.2, 2.0) * rh / 0.005
        dv = {"still": 0 * d, "approach": -d + 0.1 * e, "recede": d + 0.1 * e, "tangent": e + 1e-6 * d}[kind]
        r += [x, x + sep * d]
        v += [w, w + speed * dv]
        gm += list(IC.GU * m[k])
    gm, r, v = np.array(gm), np.array(r), np.array(v)
    radius = (3 * gm / IC.GU / (4 * np.pi * IC.RHO_3GCC)) ** (1 / 3)
    rhill = np.repeat(a, 2) * (gm / IC.GMCB / 3) ** (1 / 3)
    return IC.sort_for_integrator({"rh": r, "vh": v, "Gmass": gm, "radius": radius, "rhill": rhill}, "SYMBA")


@pytest.mark.parametrize("kind", ["still", "approach", "recede", "tangent"])
def test_recursion_decisions_bits(ctx, kind):
    pl = _pairs(kind)
    cb = {"Gmass": IC.GMCB, "radius": IC.RCB}
    g = NBodySystem(ctx, "SYMBA", cb, pl, None, dt=0.005, rhscale=1.0, precision="FP64")
    o = O.OracleSystem("SYMBA", cb, pl, None, dt=0.005, rhscale=1.0)
    for _ in range(3):
        g.step(1)
        o.step(1)
        a, b = g.get_pl(), o.get_pl()
        assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1]) and np.array_equal(a[2], b[2])
    assert g.stats()["recursion_substeps"] > 3
    g.close()
