"""The bounds-checked build (see test_bounds_checked_gpu.py) for mdot_kernel where
products outside a solve take other kernels: batches, their edges within and
across tiles, listed close pairs above a wall, ragged pairs of sources, FP64 tiles
of four CTAs, rows of a rank; and the unordered-pair kernel at the sizes that
mdot_kernel has.  In a subprocess that loads that build: every result against the
FP64 oracle, every status word clear.
"""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

SCRIPT = r"""
import json, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from libmobility_gb300 import NBody, _capi
from oracle import oracle as orc
lib = _capi.load()
assert "checked" in str(_capi.LIB_PATH)
for w in range(3):
    lib.lmg_internal_bounds_status(w, 1)
worst = {"float": 0.0, "double": 0.0}
rng = np.random.default_rng(9)
# mdot_kernel; the pairs (their warps capped far above what there are)
for mode, warps, sizes in ((1, 0, ((300, 100), (1000, 250), (33, 11), (640, 128), (777, 259),
                                   (1998, 333), (700, 7), (2600, 1300), (2049, 2049))),
                           (0, 1000000, ((1, 1), (9, 9), (16, 16), (400, 2), (700, 7)))):
    assert lib.lmg_internal_sym_override(mode, warps) == 0
    for prec in ("float", "double"):
        for wall in (0, 1):
            for ang in (0, 1):
                for N, nper in sizes:
                    p = rng.uniform(0, (nper * 4 * np.pi / 3 / 0.15) ** (1 / 3) + 1, (N, 3))
                    if wall:
                        p[:, 2] = rng.uniform(0.5, 10, N)
                    if nper > 10:
                        p[4] = p[5]
                    F = rng.normal(size=(N, 3))
                    T = rng.normal(size=(N, 3)) if ang else None
                    dt = np.float32 if prec == "float" else np.float64
                    p, F, T = (None if x is None else x.astype(dt) for x in (p, F, T))
                    s = NBody("open", "open", "single_wall" if wall else "open", precision=prec)
                    s.setParameters("advise", N // nper, nper, wallHeight=0.0 if wall else None)
                    s.initialize(viscosity=1.0, hydrodynamicRadius=1.0, includeAngular=bool(ang),
                                 tolerance=1e-4)
                    s.setPositions(p)
                    for f, t in ((F, T),) + (((F, None), (None, T)) if ang else ()):
                        out = s.Mdot(f, t)
                        ref = orc.mdot(p, f, t, a=1.0, viscosity=1.0, wall=wall,
                                       include_angular=ang, nper_batch=nper)
                        rows = s.Mdot_rows(N // 3, N // 3 + max(1, N // 2), f, t)
                        for x, y, r in zip(out, ref, rows):
                            if x is None:
                                continue
                            top = np.abs(y).max()
                            y3 = np.asarray(y).reshape(-1, 3)
                            err = max(np.abs(x - y3).max(),
                                      np.abs(r - y3[N // 3:N // 3 + max(1, N // 2)]).max())
                            worst[prec] = max(worst[prec], float(err / top))
                    if nper > 100:
                        s.sqrtMdotW_noise(rng.normal(size=(6 if ang else 3) * N))
lib.lmg_internal_sym_override(0, 0)
status = [int(lib.lmg_internal_bounds_status(w, 0)) for w in range(3)]
print(json.dumps({"worst": worst, "status": status}))
"""


def test_checked_build_runs_clean(cuda, oracle):
    from libmobility_gb300 import _build
    lib = _build.build(checked=True)
    env = dict(os.environ, LIBMOBILITY_GB300_LIB=str(lib))
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(ROOT)], env=env, capture_output=True,
                       text=True, timeout=900)
    assert r.returncode == 0, r.stdout + r.stderr
    out = json.loads(r.stdout.strip().splitlines()[-1])
    assert out["status"] == [0, 0, 0], out
    assert out["worst"]["float"] <= 1e-5 and out["worst"]["double"] <= 1e-12, out
