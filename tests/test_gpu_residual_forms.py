"""The FP32 operator in its two forms, a thread a cell and the march over planes that
large levels with cross terms take, against the FP64 operator (which the parity tests
hold to the reference's matrix).  An FP32 row rounds its 24 products and sums: 2e-6 of
the largest weight times the largest value, as in the level checks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,distort,per", [((5, 4, 6), True, (0, 0, 0)), ((30, 33, 9), True, (1, 0, 1)),
                                               ((62, 21, 17), False, (0, 0, 1)), ((63, 8, 8), False, (1, 1, 0)),
                                               ((166, 158, 160), True, (0, 0, 0)), ((160, 166, 158), True, (1, 1, 1))])
def test_apply_f32(cells, distort, per):
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300.solver import PoissonContext
    body = [] if any(per) else [(0.5, 0.5, 0.5, 0.2)]
    P = W.make_problem(cells, (1.0, 1.0, 1.0), 0.0 if per[1] else 1.0, distort, per, body, nlevels=1)
    ctx = PoissonContext().setup(P)
    try:
        x = np.random.default_rng(2).standard_normal(ctx.shapes[0]).astype(np.float32)
        y = ctx.apply(0, x.astype(np.float64))
        big = max(np.abs(w).max() for w in ctx.weights(0))
        assert np.abs(ctx.apply_f32(0, x) - y).max() <= 2e-6 * big * np.abs(x).max() * 4
    finally:
        ctx.close()
