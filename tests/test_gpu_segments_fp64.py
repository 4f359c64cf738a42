"""FP64 line solves of 33 to 64 rows, four lines a warp (segment_lines_solve), against
the relaxation with one thread per line, whose recurrences run row by row: each forced
on the finest level by a tuning file in a process of its own.  Both solves are the same
up to rounding, which grows by the condition number (below 1e6): 1e-10 of the pressure
(rtol 1e-8), after the same number of iterations."""
import json
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RUN = """
import json, sys
import numpy as np
from curvib_old_gb300 import _lib
from curvib_old_gb300 import workload as W
from curvib_old_gb300.solver import PoissonContext
cells, distort, nl, out = json.loads(sys.argv[1])
P = W.make_problem(cells, (1.0, 1.0, 1.0), 1.0, distort, (False,) * 3, [(0.5, 0.5, 0.5, 0.2)], nlevels=nl,
                   semi=(0, cells[1] % 2, 0))
ctx = PoissonContext().setup(P)
uc, _, _ = ctx.volume_flux_rev(P.ucont)
b, _ = ctx.poisson_rhs(uc, 1e-3, 1.0)
phi, st = ctx.solve(b, precision=_lib.FP64, rtol=1e-8)
np.savez(out, phi=phi, it=st["iterations"], form=ctx.tuning()["line_sweep"][-1]["zebra_f64"]["choice"])
"""


@pytest.mark.parametrize("rows,nl", [(33, 5), (40, 4), (64, 4)])
@pytest.mark.parametrize("distort", [False, True])
@pytest.mark.parametrize("form", ["split", "fused"])
def test_segments_match_row_by_row(rows, nl, distort, form, tmp_path):
    cells, got = [64, rows, 304], {}
    tiles = [1.0, 2.0] if form == "split" else [2.0, 1.0]
    for name, us in (("lines", 0.1), (form, 0.0)):
        tune, out = tmp_path / f"{name}.txt", tmp_path / f"{name}.npz"
        with open(tune, "w") as f:
            for c32, c64 in ((0, 0), (1, 1)):
                key = [c + 2 for c in cells] + [0, 0, 0, c32, c64]
                f.write(" ".join(str(v) for v in key + [2.0, 1.0, 2.0, 1.0, 1.0, 2.0] + tiles + [0.0] * 5 + [us]) + "\n")
        subprocess.run([sys.executable, "-c", RUN, json.dumps([cells, distort, nl, str(out)])], check=True, timeout=300,
                       cwd=Path(__file__).resolve().parents[1], env=dict(os.environ, CVB_TUNE_FILE=str(tune)))
        got[name] = np.load(out)
        assert str(got[name]["form"]) == name
    a, b = got["lines"]["phi"], got[form]["phi"]
    assert int(got["lines"]["it"]) == int(got[form]["it"])
    assert np.linalg.norm(a - b) <= 1e-10 * np.linalg.norm(b)
