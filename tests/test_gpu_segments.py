"""FP64 line solves of 33 to 64 rows, four lines a warp: the FP64 solve against the
mixed one, whose FP32 V-cycles solve their lines in another way.  After three
iterations the pressures differ by the FP32 cycles' rounding alone, 1e-7 of the
pressure grown by at most 1e3 (a wrong row changes the third digit).  Rows at both
ends of the range and between, lines that leave tiles part full, with and without
cross terms, periodic rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("distort,per", [(True, (0, 0, 0)), (False, (0, 0, 0)), (False, (1, 0, 1)), (True, (0, 1, 0))])
@pytest.mark.parametrize("rows", [33, 40, 47, 63, 64])
def test_fp64_matches_mixed(rows, distort, per):
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300.solver import PoissonContext
    P = W.make_problem((14, rows, 10), (1.0, 1.0, 1.0), 0.0 if per[1] else 1.0, distort, per,
                       [] if any(per) else [(0.5, 0.5, 0.5, 0.2)], nlevels=2, semi=(0, 1, 0))
    ctx = PoissonContext().setup(P)
    try:
        uc, _, _ = ctx.volume_flux_rev(P.ucont)
        b, _ = ctx.poisson_rhs(uc, 1e-3, 1.0)
        b = W.noisy_rhs(b, P.nvert, P.metrics[-1]["Aj"], 1e-3, seed=9)
        phi, st = {}, {}
        for precision in (0, 1):
            phi[precision], st[precision] = ctx.solve(b, check=False, precision=precision, rtol=1e-30, max_it=3)
        assert st[0]["iterations"] == st[1]["iterations"] == 3
        assert np.linalg.norm(phi[0] - phi[1]) <= 1e-4 * np.linalg.norm(phi[0])
    finally:
        ctx.close()
