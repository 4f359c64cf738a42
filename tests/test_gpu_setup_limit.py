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
