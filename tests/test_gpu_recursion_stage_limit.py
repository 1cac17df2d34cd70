"""The SyMBA recursion with lists of the longest length that its shared-memory stage holds and one
entry more (symba_dev.cuh rec_stage_bytes): the oracle's bits in both forms."""
import numpy as np
import pytest

from oracle import oracle as O
from swiftest_gb300 import initial_conditions as IC
from swiftest_gb300.api import Ensemble, NBodySystem

pytestmark = pytest.mark.gpu

DT = 0.002
CB = {"Gmass": IC.GMCB, "radius": IC.RCB}


def _ring(npl, entries):
    """A ring and the RHSCALE at which its first step lists that many pl-pl pairs."""
    _, pl, _ = IC.make_system(seed=11, npl=npl, ntp=0, amin=0.95, amax=1.05, mmin=1e-8, mmax=1e-6)
    pl = IC.sort_for_integrator(pl, "SYMBA")
    lo, hi = 1.0, 20.0
    for _ in range(60):
        mid = 0.5 * (lo + hi)
        n = len(O.encounter_plpl(pl["rh"], pl["vh"], pl["rhill"] * mid, DT)[0])
        if n == entries:
            return pl, mid
        lo, hi = (mid, hi) if n < entries else (lo, mid)
    raise AssertionError("no such list")


@pytest.mark.parametrize("entries", [544, 545])
def test_single(ctx, entries):
    pl, rhscale = _ring(300, entries)
    gpu = NBodySystem(ctx, "SYMBA", CB, pl, None, dt=DT, rhscale=rhscale)
    ref = O.OracleSystem("SYMBA", CB, pl, None, dt=DT, rhscale=rhscale)
    gpu.step(1)
    ref.step(1)
    assert len(gpu.plpl_list()[0]) == entries
    for a, b in zip(gpu.plpl_list() + gpu.get_pl(), ref.plpl_list() + ref.get_pl()):
        assert np.array_equal(a, b)
    gpu.close()


@pytest.mark.parametrize("entries", [217, 218])
def test_ensemble(ctx, entries):
    pl, rhscale = _ring(200, entries)
    few = {k: v[:20] for k, v in pl.items()}
    parts = [few, pl]
    E = {"integrator": "SYMBA", "dt": DT, "rhscale": rhscale, "npl": np.array([20, 200], np.int32),
         "ntp": np.zeros(2, np.int32), "GMcb": np.full(2, IC.GMCB), "Rcb": np.full(2, IC.RCB),
         "pl": {f: np.concatenate([p[f] for p in parts]) for f in ("rh", "vh", "Gmass", "radius", "rhill")},
         "tp": {f: np.zeros((0, 3)) for f in ("rh", "vh")}}
    ens = Ensemble(ctx, E, precision="FP64")
    ens.step(1)
    assert len(ens.plpl_list(1)[0]) == entries
    for s, p in enumerate(parts):
        ref = O.OracleSystem("SYMBA", CB, p, None, dt=DT, rhscale=rhscale)
        ref.step(1)
        a, b = ens.poff[s], ens.poff[s + 1]
        for x, y in zip(ens.plpl_list(s) + tuple(v[a:b] for v in ens.get_pl()), ref.plpl_list() + ref.get_pl()):
            assert np.array_equal(x, y)
    ens.close()
