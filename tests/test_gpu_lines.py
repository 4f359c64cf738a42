"""The FP64 zebra relaxation with one thread per line (kernels_lines.cu).

Whether a level takes it is the set-up autotuner's choice by time; here the
choice is made by a tuning file, in a process of its own each time.  A half-
sweep of either form is the same update up to rounding, and a solve damps the
differences, so both solves of the same right-hand side stop after the same
number of iterations, their pressures within 1e-10 of each other (rtol 1e-8:
rounding of 1e-16 grows by the condition number, below 1e6 here)."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SOLVE = """
import sys
import numpy as np
from curvib_old_gb300 import _lib
from curvib_old_gb300 import workload as W
from curvib_old_gb300.solver import PoissonContext
name, out = sys.argv[1:]
P = {
    # 7-point: two tiles a plane, the second with a few lines; 16, 20 and 88 rows (steps of eight)
    "channel68x16x152": lambda: W.config1_problem((68, 16, 152), nlevels=3),
    "channel72x88x152": lambda: W.config1_problem((72, 88, 152), nlevels=4),
    # 19-point, with a body
    "box72x20x152": lambda: W.make_problem((72, 20, 152), (1.0, 1.0, 1.0), 1.0, True, (False,) * 3,
                                           [(0.5, 0.5, 0.5, 0.2)], nlevels=3),
    # 7-point, walls and a body; one full tile a plane
    "box64x16x304": lambda: W.make_problem((64, 16, 304), (1.0, 1.0, 1.0), 1.0, False, (False,) * 3,
                                           [(0.5, 0.5, 0.5, 0.2)], nlevels=4),
}[name]()
ctx = PoissonContext().setup(P)
form = ctx.tuning()["line_sweep"][-1]["zebra_f64"]["choice"]
uc, _, _ = ctx.volume_flux_rev(P.ucont)
b, _ = ctx.poisson_rhs(uc, 1e-3, 1.0)
phi, st = ctx.solve(b, precision=_lib.FP64, rtol=1e-8)
np.savez(out, phi=phi, it=st["iterations"], form=form)
"""


@pytest.mark.parametrize("name", ["channel68x16x152", "channel72x88x152", "box72x20x152", "box64x16x304"])
def test_line_form_agrees(name, tmp_path):
    cells = [int(v) for v in name.lstrip("chanelbox").split("x")]
    per = (1, 0, 1) if name.startswith("channel") else (0, 0, 0)
    got = {}
    for form, us in (("lines", 0.1), ("split", 0.0)):
        tune = tmp_path / f"{form}.txt"
        # mx my mz px py pz cross32 cross64, then 13 timings that choose the two-kernel forms, and the lines'
        with open(tune, "w") as f:
            for c32, c64 in ((0, 0), (1, 1)):
                key = [c + 2 for c in cells] + list(per) + [c32, c64]
                f.write(" ".join(str(v) for v in key + [2.0, 1.0, 2.0, 1.0, 1.0, 2.0, 1.0, 2.0] + [0.0] * 5 + [us])
                        + "\n")
        out = tmp_path / f"{form}.npz"
        subprocess.run([sys.executable, "-c", SOLVE, name, str(out)], check=True, timeout=300,
                       cwd=Path(__file__).resolve().parents[1], env=dict(os.environ, CVB_TUNE_FILE=str(tune)))
        got[form] = np.load(out)
        assert str(got[form]["form"]) == form
    a, b = got["lines"]["phi"], got["split"]["phi"]
    assert int(got["lines"]["it"]) == int(got["split"]["it"])
    assert np.linalg.norm(a - b) <= 1e-10 * np.linalg.norm(b)
