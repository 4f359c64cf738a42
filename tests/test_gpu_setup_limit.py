"""A set-up under a device limit: the coarsest inverse's temporaries count towards it as
the matrix, two columns and the pivot tables, and for a block of up to 384 unknowns not
at all, so a context sets up with no more room than that beside what it keeps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(6, 8, 8), (5, 7, 11), (9, 10, 11)])
def test_inverse_at_the_limit(cells):
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300._lib import STATUS_NAMES, CvbError
    from curvib_old_gb300.solver import PoissonContext
    P = W.make_problem(cells, (1.0, 1.0, 1.0), 1.0, True, (False,) * 3, [], nlevels=1)
    m = int(np.prod(cells))
    free, full = PoissonContext().setup(P), PoissonContext()
    try:
        kept = free.device_bytes()
        room = 8 * (m * m + 2 * m) + 4 * (2 * m + 1) if m > 384 else 0
        if room:
            full.set_device_limit(kept + room - 1)
            with pytest.raises(CvbError) as e:
                full.setup(P)
            assert STATUS_NAMES[e.value.status] == "OOM"
        full.set_device_limit(kept + room)
        full.setup(P)
        assert full.device_bytes() == kept
        full.set_device_limit(0)  # room for the basis
        b = np.zeros(P.nvert.shape)
        b[1:-1, 1:-1, 1:-1] = np.random.default_rng(5).standard_normal(cells[::-1])
        assert np.array_equal(full.solve(b)[0], free.solve(b)[0])
    finally:
        free.close()
        full.close()


def test_a_smaller_inverse_takes_less():
    """A body that blocks coarse cells leaves a smaller inverse, and no more memory than
    a context set up with it holds."""
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300.solver import PoissonContext
    P = W.make_problem((24, 16, 20), (1.0, 1.0, 1.0), 2.0, True, (False,) * 3, [], nlevels=2)
    ctx = PoissonContext().setup(P)
    try:
        for r in (0.45, 0.2, 0.45):
            P.nvert = W.sphere_nvert(P.metrics[-1]["Cent"], [(0.5, 0.5, 0.5, r)])
            ctx.set_nvert(P.nvert)
            fresh = PoissonContext().setup(P)
            try:
                assert ctx.device_bytes() == fresh.device_bytes()
            finally:
                fresh.close()
    finally:
        ctx.close()


def test_a_set_nvert_without_room_for_its_inverse():
    """set_nvert that fails on the inverse leaves a context that solves without one (the
    coarsest level smoothed), and sets up again once there is room."""
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300._lib import STATUS_NAMES, CvbError
    from curvib_old_gb300.solver import PoissonContext
    P = W.make_problem((24, 16, 20), (1.0, 1.0, 1.0), 2.0, True, (False,) * 3, [], nlevels=2)
    small, large = (W.sphere_nvert(P.metrics[-1]["Cent"], [(0.5, 0.5, 0.5, r)]) for r in (0.2, 0.45))
    P.nvert = large
    ctx = PoissonContext().setup(P)
    P.nvert = small
    fresh = PoissonContext().setup(P)
    try:
        uc, _, _ = fresh.volume_flux_rev(P.ucont)
        b, _ = fresh.poisson_rhs(uc, 1e-3, 1.0)
        ctx.solve(b, check=False, max_it=3)  # the basis
        ctx.set_device_limit(ctx.device_bytes() + 72 * P.nvert.size)  # the operators', not the larger inverse
        with pytest.raises(CvbError) as e:
            ctx.set_nvert(small)
        assert STATUS_NAMES[e.value.status] == "OOM"
        phi, st = ctx.solve(b, check=False, max_it=3)
        assert st["iterations"] == 3 and np.isfinite(phi).all()
        ctx.set_device_limit(0)
        ctx.set_nvert(small)
        assert np.array_equal(ctx.solve(b)[0], fresh.solve(b)[0])
    finally:
        ctx.close()
        fresh.close()
