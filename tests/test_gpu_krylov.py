"""The solver's vector kernels through whole solves: bases below, at and beyond
the eight vectors a pass takes, restarts of one, sizes that leave remainders of
every block and unroll, both precisions of the basis, and a right-hand side that
the range projection changes."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[((8, 8, 8), 2), ((18, 22, 30), 2), ((48, 44, 92), 3)], ids=str)
def problem(request):
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300.solver import PoissonContext
    cells, nl = request.param
    P = W.make_problem(cells, (1.0, 1.0, 1.0), 1.0, True, (False,) * 3, [(0.5, 0.5, 0.5, 0.2)], nlevels=nl)
    L = O.levels_for(P)[-1]
    uc, _, _ = O.volume_flux_rev(L, P.ucont)
    out = O.poisson_rhs(L, uc, 1e-3, 1.0)
    b = out[0] if isinstance(out, tuple) else out
    ctx = PoissonContext().setup(P)
    yield ctx, P, L, O.lhs_csr(L), b
    ctx.close()


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("restart", [1, 7, 8, 9, 20])
def test_restarts(problem, restart, precision):
    """The reported residual is that of the returned pressure: both within the
    tolerance, which a residual's own rounding (below 1e-13 of |b| here) cannot
    move by half.  One relaxation sweep, so that long bases are filled."""
    ctx, P, L, A, b = problem
    rtol = 1e-9
    phi, st = ctx.solve(b, precision=precision, rtol=rtol, max_it=600, restart=restart, smoother=0, pre_sweeps=1,
                        post_sweeps=0)
    assert st["status"] == 0 and st["rel_residual"] <= rtol
    assert abs(st["rhs_norm"] - np.linalg.norm(b)) <= 1e-10 * np.linalg.norm(b)
    assert np.linalg.norm(b.ravel() - A @ phi.ravel()) <= 1.5 * rtol * np.linalg.norm(b)
    if restart == 20 and b.size > 10000:
        assert st["iterations"] > 9, st


@pytest.mark.parametrize("precision", [0, 1])
def test_projected_right_hand_side(problem, precision):
    """b + aj c has c removed again: sums of n terms by trees and here by numpy
    differ by far less than 1e-10 of the terms' size."""
    ctx, P, L, A, b = problem
    fluid = (L.nvert < 0.1)
    for ax in range(3):
        for end in (0, -1):
            sl = [slice(None)] * 3
            sl[ax] = end
            fluid[tuple(sl)] = False
    aj = np.asarray(P.metrics[-1]["Aj"])
    c = 3.0 * np.abs(b[fluid] / aj[fluid]).max() + 1.0
    off = b + np.where(fluid, aj * c, 0.0)
    mean = (off[fluid] / aj[fluid]).mean()
    phi, st = ctx.solve(off, precision=precision, rtol=1e-9, max_it=100, project_rhs=1)
    assert st["status"] == 0
    assert abs(st["rhs_projected"] - mean) <= 1e-10 * abs(mean)
    r = off - np.where(fluid, aj * mean, 0.0)
    assert abs(st["rhs_norm"] - np.linalg.norm(r)) <= 1e-9 * np.linalg.norm(off)
