"""The cache file of the mixed kicks' shapes (autotune.cu): a value that is no shape of its key, from a
damaged line or another version of the package, counts as not cached."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
RUN = """
import hashlib, sys
import numpy as np
sys.path.insert(0, {root!r})
from swiftest_gb300 import initial_conditions as IC
from swiftest_gb300.api import Context, Ensemble
ctx = Context(0)
for name in ("C3", "C4"):  # looks up kick_tp; kick_pl_rad and kick_tp
    E = IC.make_ensemble(name, nsys=4, scale=0.1, tp_per_pl=2)
    e = Ensemble(ctx, E, precision="MIXED", gmtiny=float(np.median(E["pl"]["Gmass"])) if name == "C4" else 0.0)
    for f in (e.set_kick_tile, e.set_kick_strip, e.set_kick_warps, e.set_kick_group):
        f(128 if f == e.set_kick_tile else 1)  # the symmetric kernel's shapes differ in rounding
    e.step(2)
    h = hashlib.sha1()
    for a in e.get_pl() + e.get_tp():
        h.update(a.tobytes())
    print(h.hexdigest())
"""


def _run(cache):
    r = subprocess.run([sys.executable, "-c", RUN.format(root=str(ROOT))], check=True, capture_output=True, text=True,
                       timeout=300, env=dict(os.environ, SWG_TUNE_CACHE=str(cache)))
    return r.stdout.split()


def test_foreign_values(ctx, tmp_path):
    cache = tmp_path / "tune.txt"
    first = _run(cache)  # timed and written
    keys = [line.split()[0] for line in cache.read_text().splitlines()]
    assert any("kick_tp" in k for k in keys) and any("kick_pl" in k for k in keys)
    for value in (5, 300, 100000):
        cache.write_text("".join(f"{k} {value}\n" for k in keys))
        assert _run(cache) == first
        # timed again and appended, so that the next run finds a shape
        last = dict(line.split() for line in cache.read_text().splitlines())
        assert all(0 <= int(v) < 5 for v in last.values())
