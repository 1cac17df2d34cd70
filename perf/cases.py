"""The work a user of this framework has it do, as cases that can be timed.

Whole calls: step loops of one system and of ensembles (WHM, HELIO, SyMBA; FP64 and mixed
precision) that end with a read-back of the state, as a run's output cadence has it.  Single
procedures: the pair kick, the Kepler drift and the encounter checks, called by an
integrator that keeps its own loop.  Sizes and distributions are those of the package's
configurations (``swiftest_gb300.initial_conditions``) and of its benchmarks.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from swiftest_gb300 import _lib as L
from swiftest_gb300 import initial_conditions as ic
from swiftest_gb300.api import Context, Ensemble, NBodySystem

PREC = {"FP64": L.SWG_FP64, "MIXED": L.SWG_MIXED}
PAIR_FLOPS = 20      # one ordered pair of a kick
DRIFT_FLOPS = 150    # one body's Kepler drift
PAIRTEST_FLOPS = 10  # one pair of an encounter check

# distributions: the configurations' (initial_conditions.CONFIGS, ENSEMBLES) and the standalone kick's
DISK = {"HELIO": dict(mmin=1e-10, mmax=1e-6, amin=0.5, amax=5.0, sig_e=0.01, sig_i=0.005),
        "WHM": dict(mmin=1e-10, mmax=1e-6, amin=0.5, amax=5.0, sig_e=0.01, sig_i=0.005),
        "SYMBA": dict(mmin=1e-10, mmax=1e-6, amin=0.3, amax=3.0, sig_e=0.01, sig_i=0.005),
        "DISK": dict(mmin=1e-11, mmax=1e-7, amin=0.5, amax=2.0, sig_e=0.02, sig_i=0.02),
        "KICK": dict(mmin=1e-12, mmax=1e-8, amin=0.5, amax=5.0, sig_e=0.01, sig_i=0.005)}
DT = {"HELIO": 0.01, "WHM": 0.01, "SYMBA": 0.005, "DISK": 0.002}
RHSCALE = {"HELIO": 6.5, "WHM": 6.5, "SYMBA": 1.0, "DISK": 1.0}


def listed():
    return [
        # a small planetary system, default precision: kernels of a few blocks, launches count
        {"name": "helio_one_small", "kind": "one", "integrator": "HELIO", "precision": "FP64", "npl": 100,
         "ntp": 1000, "steps": 20},
        # one planetesimal disk with test particles and close encounters, either precision
        {"name": "symba_one_mixed", "kind": "one", "integrator": "SYMBA", "precision": "MIXED", "npl": 2000,
         "ntp": 10000, "steps": 4},
        {"name": "symba_one_fp64", "kind": "one", "integrator": "SYMBA", "precision": "FP64", "npl": 2000,
         "ntp": 10000, "steps": 2},
        # a study of many disks at once: the framework's headline, and a part of it in FP64
        {"name": "symba_ens_mixed", "kind": "ens", "integrator": "SYMBA", "dist": "DISK", "precision": "MIXED",
         "nsys": 256, "nmin": 500, "nmax": 5000, "tp_per_pl": 0, "steps": 4},
        {"name": "symba_ens_fp64", "kind": "ens", "integrator": "SYMBA", "dist": "DISK", "precision": "FP64",
         "nsys": 24, "nmin": 500, "nmax": 5000, "tp_per_pl": 0, "steps": 1},
        # many small systems with test particles, no close encounters
        {"name": "helio_ens_mixed", "kind": "ens", "integrator": "HELIO", "dist": "HELIO", "precision": "MIXED",
         "nsys": 512, "nmin": 10, "nmax": 2000, "tp_per_pl": 5, "steps": 4},
        {"name": "whm_ens_fp64", "kind": "ens", "integrator": "WHM", "dist": "WHM", "precision": "FP64",
         "nsys": 64, "nmin": 10, "nmax": 2000, "tp_per_pl": 5, "steps": 2},
        # the single procedures, for an integrator that keeps its own loop: host arrays for the
        # kick (numpy in, numpy out), device arrays for the drift and the checks
        {"name": "kick_pl_fp64", "kind": "kick_pl", "precision": "FP64", "npl": 16384, "rad": True},
        {"name": "kick_pl_mixed", "kind": "kick_pl", "precision": "MIXED", "npl": 65536, "rad": True},
        {"name": "kick_tp_fp64", "kind": "kick_tp", "precision": "FP64", "npl": 2047, "ntp": 65537},
        {"name": "drift_large", "kind": "drift", "n": 1000003, "dt": 0.01},
        {"name": "encounter_pltp", "kind": "encounter", "mode": "TRIANGULAR", "npl": 4096, "ntp": 40001,
         "dt": 0.005},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one", "one", "one", "ens", "ens", "ens", "kick_pl", "kick_tp", "drift", "encounter"])
    prec = rng.choice(["FP64", "MIXED"])
    if kind == "one":
        integ = rng.choice(["HELIO", "SYMBA", "SYMBA", "WHM"])
        npl = _log(rng, 8, 2500)
        return {"kind": kind, "integrator": integ, "precision": prec, "npl": npl, "ntp": _log(rng, 1, 6 * npl),
                "steps": rng.randint(1, 8)}
    if kind == "ens":
        integ, dist, tpp = rng.choice([("SYMBA", "DISK", 0), ("HELIO", "HELIO", 5), ("WHM", "WHM", 5)])
        return {"kind": kind, "integrator": integ, "dist": dist, "precision": prec,
                "nsys": _log(rng, 4, 256 if prec == "MIXED" else 24), "nmin": 500 if tpp == 0 else 10,
                "nmax": _log(rng, 600, 5000 if tpp == 0 else 2000), "tp_per_pl": tpp, "steps": rng.randint(1, 4)}
    if kind == "kick_pl":
        return {"kind": kind, "precision": prec, "npl": _log(rng, 100, 65536 if prec == "MIXED" else 16384),
                "rad": rng.random() < 0.5}
    if kind == "kick_tp":
        npl = _log(rng, 10, 8192)
        return {"kind": kind, "precision": prec, "npl": npl, "ntp": _log(rng, 100, min(100000, int(1.3e8 / npl)))}
    if kind == "drift":
        return {"kind": kind, "n": _log(rng, 1000, 1000000), "dt": rng.choice([0.002, 0.005, 0.01, 0.05])}
    return {"kind": kind, "mode": rng.choice(["TRIANGULAR", "SORTSWEEP"]), "npl": _log(rng, 100, 8192),
            "ntp": _log(rng, 1000, 50000), "dt": rng.choice([0.002, 0.005, 0.01])}


# ------------------------------------------------------------------ inputs
def _sizes(case):
    """Per-system massive-body counts, log-uniform, the same for every seed (the plan's shape)."""
    return ic.ensemble_sizes(case["nsys"], case["nmin"], case["nmax"], 0)


def _system(case, seed, npl, ntp, dist):
    cb, pl, tp = ic.make_system(seed=seed, npl=int(npl), ntp=int(ntp), **DISK[dist])
    return cb, ic.sort_for_integrator(pl, case["integrator"]), tp


def _ensemble_inputs(case, seed):
    npl = _sizes(case)
    ntp = (npl * case["tp_per_pl"]).astype(np.int32)
    parts = [_system(case, seed * 1000003 + s, npl[s], ntp[s], case["dist"]) for s in range(case["nsys"])]
    pl = {k: np.concatenate([p[1][k] for p in parts]) for k in ("rh", "vh", "Gmass", "radius", "rhill")}
    tp = {k: np.concatenate([p[2][k] for p in parts]) for k in ("rh", "vh")}
    return {"integrator": case["integrator"], "dt": DT[case["dist"]], "rhscale": RHSCALE[case["dist"]], "npl": npl,
            "ntp": ntp, "GMcb": np.full(len(npl), ic.GMCB), "Rcb": np.full(len(npl), ic.RCB), "pl": pl, "tp": tp}


def _pinned(n):
    return torch.empty((n, 3), dtype=torch.float64, pin_memory=True).numpy()


_ctx = None


def _context():
    """The program's one context (a stream and its workspaces)."""
    global _ctx
    if _ctx is None:
        _ctx = Context(0)
    return _ctx


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    ctx, kind = _context(), case["kind"]
    if kind in ("one", "ens"):
        if kind == "one":
            cb, pl, tp = _system(case, seed, case["npl"], case["ntp"], case["integrator"])
            s = NBodySystem(ctx, case["integrator"], cb, pl, tp, dt=DT[case["integrator"]],
                            rhscale=RHSCALE[case["integrator"]], precision=case["precision"])
            npl, ntp = case["npl"], case["ntp"]
        else:
            s = Ensemble(ctx, _ensemble_inputs(case, seed), precision=case["precision"])
            npl, ntp = s.NPL, s.NTP
        out = {"rh": _pinned(npl), "vh": _pinned(npl)}
        if ntp:
            out |= {"trh": _pinned(ntp), "tvh": _pinned(ntp)}
        return {"case": case, "sys": s, "out": out}
    if kind == "drift":
        _, pl, _ = ic.make_system(seed=seed, npl=case["n"], ntp=0, **DISK["KICK"])
        return {"case": case, "ctx": ctx, "mu": _dev(ic.GMCB + pl["Gmass"]), "x": _dev(pl["rh"]), "v": _dev(pl["vh"]),
                "mask": torch.ones(case["n"], dtype=torch.int32, device="cuda"),
                "iflag": torch.zeros(case["n"], dtype=torch.int32, device="cuda")}
    dist = "SYMBA" if kind == "encounter" else "KICK"
    _, pl, tp = ic.make_system(seed=seed, npl=case["npl"], ntp=case.get("ntp", 0), **DISK[dist])
    pl = ic.sort_for_integrator(pl, "SYMBA")
    if kind == "encounter":
        cap = 4 * (case["npl"] + case["ntp"])  # room for the lists, which vary from step to step
        return {"case": case, "ctx": ctx, "rpl": _dev(pl["rh"]), "vpl": _dev(pl["vh"]), "rtp": _dev(tp["rh"]),
                "vtp": _dev(tp["vh"]), "renc": _dev(pl["rhill"]), "cap": cap,
                "lists": [torch.zeros(cap, dtype=torch.int32, device="cuda") for _ in range(3)]}
    return {"case": case, "ctx": ctx, "pl": pl, "tp": tp}


# ------------------------------------------------------------------ one pass
def _p(t):
    return C.c_void_p(t.data_ptr())


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("one", "ens"):
        state["sys"].step(case["steps"])
        state["sys"].get_state_async(**state["out"])
        return state["out"]
    ctx = state["ctx"]
    if kind == "kick_pl":
        pl = state["pl"]
        return ctx.kick_getacch_int_all_tri_pl(pl["rh"], pl["Gmass"], pl["radius"] if case["rad"] else None,
                                               precision=PREC[case["precision"]])
    if kind == "kick_tp":
        return ctx.kick_getacch_int_all_tp(state["tp"]["rh"], state["pl"]["rh"], state["pl"]["Gmass"],
                                           precision=PREC[case["precision"]])
    if kind == "drift":
        ctx.check("swg_drift_all", ctx.lib.swg_drift_all(
            ctx.h, _p(state["mu"]), _p(state["x"]), _p(state["v"]), case["n"], 0, 0.0, case["dt"], _p(state["mask"]),
            _p(state["iflag"]), L.SWG_MEM_DEVICE))
        return {"x": state["x"], "v": state["v"], "iflag": state["iflag"]}
    n = C.c_int64(0)
    i1, i2, lv = state["lists"]
    mode = {"TRIANGULAR": L.SWG_ENC_TRIANGULAR, "SORTSWEEP": L.SWG_ENC_SORTSWEEP}[case["mode"]]
    ctx.check("swg_encounter_check_all_pltp", ctx.lib.swg_encounter_check_all_pltp(
        ctx.h, mode, case["npl"], case["ntp"], _p(state["rpl"]), _p(state["vpl"]), _p(state["rtp"]), _p(state["vtp"]),
        _p(state["renc"]), case["dt"], state["cap"], C.byref(n), _p(i1), _p(i2), _p(lv), L.SWG_MEM_DEVICE))
    # the program's list buffers whole: the first n entries are the list, the rest stay zero
    return {"n": n.value, "index1": i1, "index2": i2, "lvdotr": lv}


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind in ("one", "ens"):
        npl = np.array([case["npl"]]) if kind == "one" else _sizes(case).astype(np.int64)
        ntp = np.array([case["ntp"]]) if kind == "one" else npl * case["tp_per_pl"]
        pairs = float((npl * (npl - 1) + npl * ntp).sum())
        bodies = float((npl + ntp).sum())
        kicks = 1 if case["integrator"] == "WHM" else 2
        flops = case["steps"] * (kicks * PAIR_FLOPS * pairs + DRIFT_FLOPS * bodies)
        if case["integrator"] == "SYMBA":
            flops += case["steps"] * PAIRTEST_FLOPS * float((npl * (npl - 1) / 2 + npl * ntp).sum())
        return {"bytes": case["steps"] * 96 * bodies + 48 * bodies, "flops": flops}
    if kind == "kick_pl":
        n = case["npl"]
        return {"bytes": (24 + 8 + 8 * case["rad"] + 24) * n, "flops": PAIR_FLOPS * n * (n - 1)}
    if kind == "kick_tp":
        return {"bytes": 32 * case["npl"] + 52 * case["ntp"], "flops": PAIR_FLOPS * case["npl"] * case["ntp"]}
    if kind == "drift":
        return {"bytes": 112 * case["n"], "flops": DRIFT_FLOPS * case["n"]}
    return {"bytes": 56 * case["npl"] + 48 * case["ntp"], "flops": PAIRTEST_FLOPS * case["npl"] * case["ntp"]}


# ------------------------------------------------------------------ 64-bit references
def _accel(x, y, gm, same):
    """Accelerations at x (n, 3) from the bodies gm at y (m, 3), in 64 bits; same: x is y."""
    out = torch.zeros_like(x)
    step = max(1, int(4e7) // max(1, len(y)))
    for a in range(0, len(x), step):
        d = y[None, :, :] - x[a:a + step, None, :]
        r2 = (d * d).sum(2)
        if same:
            k = torch.arange(a, min(a + step, len(x)), device=x.device)
            r2[k - a, k] = math.inf
        out[a:a + step] = ((gm[None, :] / (r2 * r2.sqrt()))[:, :, None] * d).sum(1)
    return out


def _kepler(mu, x, v, dt):
    """Two-body motion of elliptic orbits over dt (difference of the eccentric anomaly by Newton)."""
    r0 = x.norm(dim=1)
    u = (x * v).sum(1)
    a = 1.0 / (2.0 / r0 - (v * v).sum(1) / mu)
    n = torch.sqrt(mu / a) / a
    ec, es = 1.0 - r0 / a, u / (n * a * a)
    dm = torch.remainder(n * dt, 2 * math.pi)
    y = dm + es * (torch.cos(dm) - 1) + ec * torch.sin(dm)
    for _ in range(12):
        s, c1 = torch.sin(y), 2 * torch.sin(0.5 * y) ** 2  # c1 = 1 - cos y
        y = y - (y - ec * s + es * c1 - dm) / (1 - ec * (1 - c1) + es * s)
    s, c1 = torch.sin(y), 2 * torch.sin(0.5 * y) ** 2
    r = 1 - ec * (1 - c1) + es * s
    f, g = 1 - (a / r0) * c1, dm / n + (s - y) / n
    fd, gd = -(a * n * s) / (r0 * r), 1 - c1 / r
    return f[:, None] * x + g[:, None] * v, fd[:, None] * x + gd[:, None] * v


def _helio(cb, pl, tp, dt, steps):
    """Democratic heliocentric kick-drift-kick steps of one system."""
    gm, x, vh = _dev(pl["Gmass"]), _dev(pl["rh"]), _dev(pl["vh"])
    y, w = _dev(tp["rh"]), _dev(tp["vh"])
    gc, h = cb["Gmass"], 0.5 * dt
    mom = lambda v: (gm[:, None] * v).sum(0)  # noqa: E731
    v = vh - mom(vh) / (gc + gm.sum())
    w = w - mom(vh) / (gc + gm.sum())
    for _ in range(steps):
        p = mom(v) / gc
        x, y = x + p * h, y + p * h
        v, w = v + _accel(x, x, gm, True) * h, w + _accel(y, x, gm, False) * h
        x, v = _kepler(gc, x, v, dt)
        if len(y):
            y, w = _kepler(gc, y, w, dt)
        v, w = v + _accel(x, x, gm, True) * h, w + _accel(y, x, gm, False) * h
        p = mom(v) / gc
        x, y = x + p * h, y + p * h
    p = mom(v) / gc
    return [t.cpu().numpy() for t in (x, v + p, y, w + p)]


def exact(case, seed):
    """Values in 64 bits, without the package's kernels: kicks, drift and HELIO steps.  WHM and
    SyMBA steps (Jacobi coordinates, recursive sub-steps) have none here, nor have the
    encounter lists, which are whole numbers."""
    kind = case["kind"]
    if kind == "kick_pl" or kind == "kick_tp":
        _, pl, tp = ic.make_system(seed=seed, npl=case["npl"], ntp=case.get("ntp", 0), **DISK["KICK"])
        pl = ic.sort_for_integrator(pl, "SYMBA")
        y, gm = _dev(pl["rh"]), _dev(pl["Gmass"])
        x = y if kind == "kick_pl" else _dev(tp["rh"])
        return _accel(x, y, gm, kind == "kick_pl").cpu().numpy()
    if kind == "drift":
        _, pl, _ = ic.make_system(seed=seed, npl=case["n"], ntp=0, **DISK["KICK"])
        x, v = _kepler(_dev(ic.GMCB + pl["Gmass"]), _dev(pl["rh"]), _dev(pl["vh"]), case["dt"])
        return {"x": x, "v": v, "iflag": None}
    if case.get("integrator") != "HELIO":
        return None
    if kind == "one":
        parts = [_system(case, seed, case["npl"], case["ntp"], "HELIO")]
    else:
        npl = _sizes(case)
        parts = [_system(case, seed * 1000003 + s, npl[s], npl[s] * case["tp_per_pl"], case["dist"])
                 for s in range(case["nsys"])]
    got = [_helio(cb, pl, tp, DT["HELIO"], case["steps"]) for cb, pl, tp in parts]
    out = dict(zip(("rh", "vh", "trh", "tvh"), (np.concatenate(g) for g in zip(*got))))
    return out
