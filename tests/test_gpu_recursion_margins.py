"""The recursion's FP32 decisions (symba_dev.cuh d_list_pair, d_collision_far) against the FP64 tests
that they stand for, on pairs at and about every threshold: the device functions are compiled
into a probe.  And whole steps of pairs about their shells and about touching, against the oracle."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from oracle import oracle as O
from swiftest_gb300 import build as B
from swiftest_gb300 import initial_conditions as IC
from swiftest_gb300.api import NBodySystem

pytestmark = pytest.mark.gpu

N = 1 << 20
OFFSETS = np.array([0.0, 2e-16, -2e-16, 1e-15, -1e-15, 1e-8, -1e-8, 1e-7, -1e-7, 1e-6, -1e-6, 4e-6, -4e-6, 1e-5, -1e-5,
                    2e-5, -2e-5, 4e-5, -4e-5, 1e-4, -1e-4, 0.1, -0.1])

PROBE = r"""
#include "symba_dev.cuh"
#include "collision_one.cuh"
using namespace swg;
using namespace swg::sdev;
// p: 12 numbers a pair; bad[0 .. 3]: decisions that differ (list: FP64, mixed path; collision), taken in FP32
__global__ void k(int n, const double *p, unsigned long long *bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double *x = p + 12 * (size_t)i, *v = x + 3;
    const double rhs1 = x[6], rhs2 = x[7], rsp = x[8], ra1 = x[9], ra2 = x[10], dt = x[11];
    const bool isp = i & 1;
    for (int fast = 0; fast < 2; fast++) {
        int lvd = -1, lvd64 = -1, le = 0;
        const bool got = d_list_pair(fast, isp, x, v, rhs1, isp ? rhs2 : 0.0, rsp, ra1, isp ? ra2 : 0.0, dt, lvd);
        const double renci = rhs1 * rsp, rcrit = isp ? renci + rhs2 * rsp : renci;
        if (fast) d_enc_one_fast(x[0], x[1], x[2], v[0], v[1], v[2], rcrit, dt, le, lvd64);
        else d_enc_one(x[0], x[1], x[2], v[0], v[1], v[2], rcrit, dt, le, lvd64);
        const double rs = isp ? ra1 + ra2 : ra1;
        if (le) le = x[0] * x[0] + x[1] * x[1] + x[2] * x[2] > rs * rs;
        if (got != (le != 0) || lvd != lvd64) atomicAdd(&bad[fast], 1ull);
    }
    for (int lv = 0; lv < 2; lv++) {
        const double rlim = isp ? ra1 + ra2 : ra1;
        if (!d_collision_far(-x[0], -x[1], -x[2], -v[0], -v[1], -v[2], rlim, dt, lv)) continue;
        atomicAdd(&bad[3], 1ull);
        if (d_collision_one(-x[0], -x[1], -x[2], -v[0], -v[1], -v[2], 1e-9, rlim, dt, lv)) atomicAdd(&bad[2], 1ull);
    }
}
extern "C" int probe(int n, const double *p, unsigned long long *bad) {
    const size_t b = sizeof(double) * 12 * (size_t)n;
    double *d;
    unsigned long long *c;
    if (cudaMalloc(&d, b) || cudaMalloc(&c, 32)) return 1;
    cudaMemcpy(d, p, b, cudaMemcpyHostToDevice);
    cudaMemset(c, 0, 32);
    k<<<(n + 127) / 128, 128>>>(n, d, c);
    cudaMemcpy(bad, c, 32, cudaMemcpyDeviceToHost);
    cudaFree(d);
    cudaFree(c);
    return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    tmp = tmp_path_factory.mktemp("probe")
    (tmp / "probe.cu").write_text(PROBE)
    subprocess.run([B.nvcc(), *B.ARCH, *B.NVFLAGS, "-I", str(B.CSRC), "-shared", "-o", str(tmp / "probe.so"),
                    str(tmp / "probe.cu")], check=True)
    lib = C.CDLL(str(tmp / "probe.so"))

    def run(p):
        bad = np.zeros(4, np.uint64)
        q = np.ascontiguousarray(p)
        assert lib.probe(len(q), q.ctypes.data_as(C.c_void_p), bad.ctypes.data_as(C.c_void_p)) == 0
        return [int(b) for b in bad]

    return run


def _unit(rng, n):
    d = rng.normal(size=(n, 3))
    return d / np.linalg.norm(d, axis=1, keepdims=True)


def _cases(kind, seed):
    """N pairs (displacement, velocity, rhill rhscale of both, shell factor, radii, dt), the scales spread
    over twelve decades, `kind`'s threshold met up to one of OFFSETS."""
    rng = np.random.default_rng(seed)
    off = lambda: 1.0 + rng.choice(OFFSETS, N)  # noqa: E731
    rc = 10.0 ** rng.uniform(-9, 3, N)
    dt = 10.0 ** rng.uniform(-6, 1, N) * rng.choice([1, 1, 1, -1], N)
    share, rsp = rng.uniform(0.05, 0.95, N), 0.48075 ** rng.integers(0, 8, N)
    share[::2] = 1.0  # the even pairs have a test particle: one body's radii
    d = _unit(rng, N)
    e = np.cross(d, _unit(rng, N))
    e /= np.linalg.norm(e, axis=1, keepdims=True)
    sep = rc * rng.uniform(0.3, 3.0, N)
    speed = 10.0 ** rng.uniform(-3, 3, N) * rc / np.abs(dt)
    radial = rng.uniform(-1, 1, N)
    rad = sep * rng.uniform(0.01, 0.9, N)
    if kind == "radius":  # at the encounter radius
        sep = rc * off()
    elif kind == "closest":  # the closest approach at the encounter radius
        sep = rc * rng.uniform(1.001, 30.0, N)
        radial = -np.sqrt(1 - np.minimum(rc / sep * off(), 1.0) ** 2)
    elif kind == "step":  # the separation at the step's end at the encounter radius
        sep = rc * rng.uniform(1.001, 3.0, N)
        radial, speed = -np.ones(N), (sep - rc * off()) / np.abs(dt)
    elif kind == "time":  # closest approach at the step's end
        radial = -rng.uniform(0.01, 1.0, N)
        speed = -radial * sep / np.abs(dt) * off()
        radial = np.where(rng.random(N) < 0.5, radial, -radial)
    elif kind == "tangent":  # almost perpendicular
        radial = rng.choice(OFFSETS, N)
    elif kind == "touch":  # overlapping or not
        rad = sep * off()
    elif kind == "crossing":  # receding bodies whose crossing time is the step
        radial, speed = rng.uniform(0.01, 1.0, N), sep / np.abs(dt) * off()
        rad = sep * rng.uniform(0.5, 0.99, N)
    elif kind == "plain":  # zero components and velocities, infinities and NaN
        d[rng.random((N, 3)) < 0.3] = 0.0
        speed *= rng.choice([0.0, 1e-20, 1.0, 1e20], N)
        sep[rng.random(N) < 0.01] = np.nan
        sep[rng.random(N) < 0.01] = np.inf
        rc[rng.random(N) < 0.05] = 0.0
        rad[rng.random(N) < 0.05] = 0.0
    x = sep[:, None] * np.where(np.isfinite(sep)[:, None], d, 1.0)
    tangential = np.sqrt(np.maximum(1 - radial ** 2, 0.0))
    v = speed[:, None] * (radial[:, None] * d + tangential[:, None] * e)
    return np.column_stack([x, v, rc * share / rsp, rc * (1 - share) / rsp, rsp, rad * share, rad * (1 - share), dt])


@pytest.mark.parametrize("kind", ["radius", "closest", "step", "time", "tangent", "touch", "crossing", "plain"])
def test_decisions(probe, kind):
    list64, mixed, collision, far = probe(_cases(kind, 7))
    assert (list64, mixed, collision) == (0, 0, 0)
    assert far > N // 20  # and most of the far pairs are decided


def _pairs(offset, touch, kind, n=16, tp=False):
    """n pairs well apart, second bodies at a shell's radius (touch: the sum of the radii, which are made
    large) times 1 + the offset, at rest, approaching, receding or almost tangential."""
    rng = np.random.default_rng(17 + len(kind))
    a = 0.4 + 0.25 * np.arange(n)
    m = 10.0 ** rng.uniform(-9, -7, (n, 2))
    th = rng.uniform(0, 2 * np.pi, n)
    r, v, gm, radius, rhill = [], [], [], [], []
    for k in range(n):
        x = a[k] * np.array([np.cos(th[k]), np.sin(th[k]), 0.0])
        w = np.sqrt(IC.GMCB / a[k]) * np.array([-np.sin(th[k]), np.cos(th[k]), 0.0])
        rh = a[k] * (m[k] / 3.0) ** (1 / 3)
        if tp:
            rh[1] = 0.0
        d, e = _unit(rng, 2)
        e = np.cross(d, e)
        e /= np.linalg.norm(e)
        sep = rh.sum() * 0.48075 ** (k % 4)
        R = 0.02 * rh  # about the physical radii
        if touch:
            R = sep * rng.uniform(0.2, 0.8) * np.array([1.0, 0.0]) if tp else sep * np.array([0.6, 0.4])
            sep = R.sum()
        sep *= 1.0 + offset
        speed = rng.uniform(0.2, 2.0) * sep / 0.005
        dv = {"still": 0 * d, "approach": -d + 0.1 * e, "recede": d + 0.1 * e, "tangent": e + 1e-6 * d}[kind]
        r += [x, x + sep * d]
        v += [w, w + speed * dv]
        gm += list(IC.GU * m[k])
        radius += list(R)
        rhill += list(rh)
    r, v, gm, radius, rhill = map(np.array, (r, v, gm, radius, rhill))
    one = slice(0, None, 2) if tp else slice(None)
    pl = IC.sort_for_integrator({"rh": r[one], "vh": v[one], "Gmass": gm[one], "radius": radius[one],
                                 "rhill": rhill[one]}, "SYMBA")
    return pl, {"rh": r[1::2], "vh": v[1::2]} if tp else None


@pytest.mark.parametrize("tp", [False, True])
@pytest.mark.parametrize("touch", [False, True])
@pytest.mark.parametrize("offset", [0.0, 1e-6, -1e-6, 1e-12, -1e-12])
@pytest.mark.parametrize("kind", ["still", "approach", "recede", "tangent"])
def test_steps(ctx, kind, offset, touch, tp):
    pl, tps = _pairs(offset, touch, kind, tp=tp)
    cb = {"Gmass": IC.GMCB, "radius": IC.RCB}
    g = NBodySystem(ctx, "SYMBA", cb, pl, tps, dt=0.005, rhscale=1.0, precision="FP64")
    o = O.OracleSystem("SYMBA", cb, pl, tps, dt=0.005, rhscale=1.0)
    for _ in range(3):
        g.step(1)
        o.step(1)
        for a, b in zip(g.get_pl() + (g.get_tp() if tp else ()), o.get_pl() + (o.get_tp() if tp else ())):
            assert np.array_equal(a, b)
        assert g.stats() == o.stats()
    assert g.stats()["recursion_substeps"] > 0
    g.close()
