"""What chooses the FP64 zebra relaxation with one thread per line: the level's shape
(lines_pay), so that a solve's bits do not depend on what else ran while the set-up
timed its kernels.  The FP64 zebra forms that are chosen by time give the same bits, and
so do the FP64 Jacobi sweep's two where both compose the same rows a lane (33 to 64)."""
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
cells, per, distort, nl, out, smoother = json.loads(sys.argv[1])
P = W.make_problem(cells, (1.0, 1.0, 1.0), 1.0, distort, per, [], nlevels=nl, semi=(0, cells[1] % 2, 0))
ctx = PoissonContext().setup(P)
r = {"choice": np.array([t[("f64", "zebra_f64")[smoother]]["choice"] for t in ctx.tuning()["line_sweep"]])}
if out:
    uc, _, _ = ctx.volume_flux_rev(P.ucont)
    b, _ = ctx.poisson_rhs(uc, 1e-3, 1.0)
    b = W.noisy_rhs(b, P.nvert, P.metrics[-1]["Aj"], 1e-3, seed=7)
    r["phi"] = ctx.solve(b, check=False, precision=_lib.FP64, rtol=1e-30, max_it=4, smoother=smoother,
                         omega=(0.85, 1.3)[smoother])[0]
    np.savez(out, **r)
print(" ".join(r["choice"]))
"""


def _run(tune, cells, per, distort, nl, out=None, smoother=1):
    import json
    job = json.dumps([cells, per, distort, nl, out and str(out), smoother])
    r = subprocess.run([sys.executable, "-c", RUN, job], check=True, timeout=300,
                       cwd=Path(__file__).resolve().parents[1], capture_output=True, text=True,
                       env=dict(os.environ, CVB_TUNE_FILE=str(tune)))
    return r.stdout.split()


def _write(path, levels, per, timings):
    """A tuning file with the same thirteen timings for every level and cross flag."""
    with open(path, "w") as f:
        for cells in levels:
            for c in (0, 1):
                f.write(" ".join(str(v) for v in [n + 2 for n in cells] + list(per) + [c, c] + timings) + "\n")


# us32[2], us64[2], zebra f32[2], zebra f64[2] (split, fused), tma, 4-line tiles
SPLIT = [2.0, 1.0, 2.0, 1.0, 1.0, 2.0, 1.0, 2.0] + [0.0] * 5
FUSED = [1.0, 2.0, 1.0, 2.0, 2.0, 1.0, 2.0, 1.0] + [0.0] * 5
LEVELS = {2: lambda c: [[n // 2 for n in c], c], 3: lambda c: [[n // 4 for n in c], [n // 2 for n in c], c]}


def test_files_without_the_fourteenth_timing_are_read(tmp_path):
    cells, per = [16, 40, 12], (0, 0, 0)
    for name, timings in (("split", SPLIT), ("fused", FUSED)):
        _write(tmp_path / name, LEVELS[2](cells), per, timings)
        before = (tmp_path / name).read_text()
        assert set(_run(tmp_path / name, cells, per, False, 2)) == {name}
        assert (tmp_path / name).read_text() == before  # nothing measured again


@pytest.mark.parametrize("cells,lines", [((64, 16, 304), True), ((72, 88, 152), False)])
def test_the_choice_is_the_shapes(cells, lines, tmp_path):
    for k, scale in enumerate((1e-3, 1e6)):  # tile kernels far faster than any, and far slower
        tune = tmp_path / str(k)
        _write(tune, LEVELS[2](list(cells)), (0, 0, 0), [scale * t for t in SPLIT])
        assert (_run(tune, cells, (0, 0, 0), False, 2)[-1] == "lines") == lines


@pytest.mark.parametrize("cells,per,distort,nl", [((16, 16, 24), (0, 0, 0), False, 2), ((24, 40, 24), (1, 0, 1), False, 3),
                                                  ((24, 80, 16), (0, 0, 0), True, 3), ((18, 144, 8), (0, 0, 0), True, 2),
                                                  ((64, 16, 304), (0, 0, 0), True, 2)])
def test_forms_chosen_by_time_give_the_same_bits(cells, per, distort, nl, tmp_path):
    got = {}
    for name, timings in (("split", SPLIT), ("fused", FUSED)):
        _write(tmp_path / name, LEVELS[nl](list(cells)), per, timings)
        assert name in _run(tmp_path / name, cells, per, distort, nl, tmp_path / f"{name}.npz")
        got[name] = np.load(tmp_path / f"{name}.npz")["phi"]
    assert np.array_equal(got["split"], got["fused"])


@pytest.mark.parametrize("rows", [33, 40, 63, 64])
@pytest.mark.parametrize("distort", [False, True])
def test_jacobi_forms_of_33_to_64_rows_give_the_same_bits(rows, distort, tmp_path):
    cells, per, got = [14, rows, 10], (0, 0, 0), {}
    for name, timings in (("split", SPLIT), ("fused", FUSED)):
        # an odd number of rows stays on the coarse level
        _write(tmp_path / name, [[7, rows, 5], cells] if rows % 2 else LEVELS[2](cells), per, timings)
        out = tmp_path / f"{name}.npz"
        assert set(_run(tmp_path / name, cells, per, distort, 2, out, smoother=0)) == {name}
        got[name] = np.load(out)["phi"]
    assert np.array_equal(got["split"], got["fused"])
