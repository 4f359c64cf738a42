"""The coarsest level's dense inverse (k_gj_panel, k_gj_update).

A hierarchy of one level is solved by the inverse alone, so FGMRES needs one
iteration, or a few where rounding leaves more than the tolerance: the inverse
is off by the unit roundoff times the matrix's condition number (below 1e5
here), so three iterations reach 1e-10.  Sizes at the edges of its panels of 8
columns and tiles of 16, 32 and 64, with a body that leaves rows out, and with face
Jacobians of random sign and size, whose rows are not diagonally dominant, so
that pivot rows move."""
import types

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(2, 2, 2), (3, 3, 3), (4, 4, 4), (5, 13, 2), (3, 8, 8), (6, 6, 6), (6, 8, 8), (7, 9, 12),
                                   (8, 8, 12), (9, 10, 11)])
@pytest.mark.parametrize("rows", ["dominant", "pivoting", "body"])
def test_one_level_solve(cells, rows):
    from curvib_old_gb300 import _lib
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300.solver import PoissonContext
    rng = np.random.default_rng(sum(cells))
    P = W.make_problem(cells, (1.0, 1.0, 1.0), 1.0, True, (False,) * 3, [], nlevels=1)
    m = dict(P.metrics[0])
    nvert = P.nvert.copy()
    if rows == "pivoting":
        for nm in ("IAj", "JAj", "KAj"):
            f = m[nm].shape
            m[nm] = m[nm] * rng.uniform(0.5, 2.0, f) * rng.choice([-1.0, 1.0], f)
    if rows == "body":
        if min(cells) < 4:
            pytest.skip("no room for a body")
        nvert[2, 2, 2] = 3.0
    Q = types.SimpleNamespace(metrics=[m], nvert=nvert, bctype=P.bctype, semi=P.semi)
    ctx = PoissonContext().setup(Q)
    try:
        b = np.zeros(nvert.shape)
        fl = np.zeros(nvert.shape, dtype=bool)
        fl[1:-1, 1:-1, 1:-1] = nvert[1:-1, 1:-1, 1:-1] < 0.1
        b[fl] = rng.standard_normal(int(fl.sum()))
        _, st = ctx.solve(b, precision=_lib.FP64, rtol=1e-10, max_it=20)
        assert st["iterations"] <= 3 and st["rel_residual"] <= 1e-10, st
        # a second set-up gives the same inverse
        p0, _ = ctx.solve(b, precision=_lib.FP64, rtol=1e-10, max_it=20)
        ctx.set_nvert(nvert)
        p1, _ = ctx.solve(b, precision=_lib.FP64, rtol=1e-10, max_it=20)
        assert np.array_equal(p0, p1)
    finally:
        ctx.close()


def test_graphs_follow_a_moving_body():
    """Captured V-cycles survive a set_nvert that leaves their kernels'
    arguments alone, and are dropped by one that does not (a body that blocks
    coarse cells): each solve equals a fresh context's, bit for bit."""
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300.solver import PoissonContext
    P = W.make_problem((24, 16, 20), (1.0, 1.0, 1.0), 2.0, True, (False,) * 3, [])
    cent = P.metrics[-1]["Cent"]
    bodies = [[], [(0.5, 0.5, 0.5, 0.08)], [(0.55, 0.5, 0.5, 0.08)], [(0.5, 0.5, 0.5, 0.45)], [(0.5, 0.5, 0.5, 0.08)]]
    ctx = PoissonContext().setup(P)
    try:
        for spheres in bodies:
            nv = W.sphere_nvert(cent, spheres)
            ctx.set_nvert(nv)
            P.nvert = nv
            fresh = PoissonContext().setup(P)
            try:
                for c in (ctx, fresh):
                    c.uc = c.volume_flux_rev(P.ucont)[0]
                    c.b = c.poisson_rhs(c.uc, 1e-3, 1.0)[0]
                    for _ in range(2):  # the second solve replays what the first captured
                        c.phi, c.st = c.solve(c.b)
                assert ctx.st["iterations"] == fresh.st["iterations"]
                assert np.array_equal(ctx.phi, fresh.phi)
            finally:
                fresh.close()
    finally:
        ctx.close()
