"""A V-cycle's small levels in the tail kernels (kernels_tail.cu) against the batch
engine, which runs the same cycle level by level: the pressures after three
iterations agree to the rounding of the cycles, FP64 1e-16 and FP32 1e-7 of the
pressure grown by what an ill-conditioned combination of three directions costs
(1e6 and 1e3 at most), where a dropped or stale neighbour changes the third digit.
Levels of one tile and of all 64, lines of 32 rows, one to three levels, with and
without cross terms, in and out of place (an odd periodic level)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = {
    # cells, periodic, semi-coarsened, distorted, levels
    "two_levels": ((32, 32, 32), (0, 0, 0), (0, 0, 0), True, 4),
    "three_levels": ((64, 64, 32), (0, 0, 0), (0, 0, 0), True, 5),
    "rows32": ((24, 64, 32), (0, 0, 0), (0, 0, 0), True, 3),
    "all_tiles": ((56, 16, 32), (0, 0, 0), (0, 0, 0), True, 3),
    "one_tile": ((8, 16, 8), (0, 0, 0), (0, 0, 0), True, 3),
    "plain": ((32, 24, 40), (1, 0, 1), (0, 0, 0), False, 4),
    "odd_periodic": ((15, 24, 24), (1, 0, 0), (1, 0, 0), False, 3),
    "odd_periodic_cross": ((24, 24, 15), (0, 0, 1), (0, 0, 1), True, 3),
    "semi": ((20, 16, 32), (0, 0, 0), (0, 1, 0), True, 3),
}


@pytest.mark.parametrize("pre,post", [(1, 0), (2, 2), (3, 1)])
@pytest.mark.parametrize("name", sorted(GRIDS))
def test_tail_matches_level_by_level(name, pre, post):
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300.solver import PoissonContext, SolveBatch
    cells, per, semi, distort, nl = GRIDS[name]
    body = [] if not distort else [(0.5, 0.5, 0.5, 0.2)]
    P = W.make_problem(cells, (1.0, 1.0, 1.0), 1.0, distort, per, body, nlevels=nl, semi=semi)
    ctx = PoissonContext().setup(P)
    try:
        uc, _, _ = ctx.volume_flux_rev(P.ucont)
        b, _ = ctx.poisson_rhs(uc, 1e-3, 1.0)
        b = W.noisy_rhs(b, P.nvert, P.metrics[-1]["Aj"], 1e-3, seed=5)
        for precision, tol in ((0, 1e-10), (1, 1e-4)):
            opts = dict(precision=precision, rtol=1e-30, max_it=3, pre_sweeps=pre, post_sweeps=post)
            for _ in range(3):  # as launched, captured, replayed
                phi, one = ctx.solve(b, check=False, **opts)
            B = SolveBatch(**opts)
            try:
                B.submit(ctx, b=b)
                while B.step():
                    pass
                (_, many), = B.poll()
                ref = ctx.get_phi()
            finally:
                B.close()
            assert one["iterations"] == many["iterations"] == 3
            assert np.linalg.norm(phi - ref) <= tol * np.linalg.norm(ref), precision
    finally:
        ctx.close()
