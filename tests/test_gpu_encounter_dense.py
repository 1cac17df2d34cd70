"""TRIANGULAR checks of one list whose bodies all lie at nearly the same radius, so that the radial
order leaves every pair to be tested (encounter_sorted.cu ONE_BLOCKS)."""
import time

import numpy as np
import pytest

from oracle import oracle as O
from swiftest_gb300 import initial_conditions as IC

pytestmark = pytest.mark.gpu


def _ring(n):
    _, pl, _ = IC.make_system(seed=n, npl=n, ntp=0, amin=1.0, amax=1.0001, sig_e=1e-3, sig_i=1e-3)
    return pl["rh"], pl["vh"], np.full(n, 1e-3)


# chunks of partners: 4, 5 and 12 sub-tiles each, the last one whole, part of one and one body
@pytest.mark.parametrize("n", [4480, 4481, 5000, 5121, 8192, 8193])
def test_ring(ctx, n):
    r, v, renc = _ring(n)
    g = ctx.encounter_check_all_plpl(r, v, renc, 0.005, cap=100000)
    o = O.encounter_plpl(r, v, renc, 0.005)
    assert len(o[0]) > 1000
    for a, b in zip(g, o):
        assert np.array_equal(a, b)


def test_ring_time(ctx):
    """A list's own pairs take no longer than those of the list against as many test particles
    (twice as many pairs, spread over the GPU's SMs by the same rule)."""
    r, v, renc = _ring(8192)

    def best(f):
        t = []
        for _ in range(15):
            t0 = time.perf_counter()
            f()
            t.append(time.perf_counter() - t0)
        return min(t)

    own = best(lambda: ctx.encounter_check_all_plpl(r, v, renc, 0.005, cap=100000))
    both = best(lambda: ctx.encounter_check_all_pltp(r, v, r, v, renc, 0.005, cap=100000))
    assert own < 1.5 * both


# below and from the count of massive bodies on with which long lists are sorted (encounter.cu SORTED_PL)
@pytest.mark.parametrize("npl", [1, 8, 63, 64])
def test_few_massive_bodies(ctx, npl):
    _, pl, tp = IC.make_system(seed=npl, npl=npl, ntp=10000000 // npl + 1 if npl > 1 else 1000, amin=0.3, amax=3.0)
    near = slice(0, len(tp["rh"]), 1 + len(tp["rh"]) // 500)
    tp["rh"][near] = pl["rh"][0] * (1 + 1e-5)
    args = pl["rh"], pl["vh"], tp["rh"], tp["vh"], 3.0 * pl["rhill"], 0.005
    g, o = ctx.encounter_check_all_pltp(*args, cap=100000), O.encounter_pltp(*args)
    assert len(o[0]) > 100
    for a, b in zip(g, o):
        assert np.array_equal(a, b)
