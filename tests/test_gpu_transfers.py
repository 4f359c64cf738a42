"""Restriction and interpolation at sizes that march one, two and four planes a
thread, with cells between fluid and blocked scattered over the box and values
at the edges of the exact integer forms: equal to the oracle's."""
import types

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu
EDGE = [0.0, -0.0, 2.0**-1022, 2.0**-1020, 5e-324, 3e-310, 2.0**1020, 1.5 * 2.0**1023, -(2.0**1019), np.inf, np.nan]



@pytest.mark.parametrize("cells,semi", [((20, 22, 18), (0, 0, 0)), ((20, 22, 18), (1, 0, 0)), ((20, 22, 18), (0, 1, 0)),
                                        ((20, 22, 18), (0, 0, 1)), ((100, 120, 110), (0, 0, 0)),
                                        ((140, 130, 150), (0, 0, 0))])
def test_transfers_match_oracle(cells, semi):
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300.solver import PoissonContext
    P = W.make_problem(cells, (1.0, 1.0, 1.0), 1.0, False, (False,) * 3, [], nlevels=2, semi=semi)
    rng = np.random.default_rng(3)
    nv = P.nvert.copy()
    at = rng.choice(nv.size, nv.size // 60, replace=False)
    nv.ravel()[at] = rng.choice([-0.0, 0.05, 0.0999, 0.5, 1.0, 3.0], at.size)
    P = types.SimpleNamespace(metrics=P.metrics, nvert=nv, ucont=P.ucont, bctype=P.bctype, semi=P.semi)
    Ls = O.levels_for(P)
    ctx = PoissonContext().setup(P)
    try:
        for l, f in ((1, lambda x: (ctx.restrict(0, x), O.restrict(Ls[1], Ls[0], x))),
                     (0, lambda x: (ctx.interpolate(1, x), O.interpolate(Ls[0], Ls[1], x)))):
            x = rng.standard_normal(ctx.shapes[l])
            with np.errstate(all="ignore"):
                assert np.array_equal(*f(x), equal_nan=True)
                at = rng.choice(x.size, x.size // 50, replace=False)
                x.ravel()[at] = rng.choice(EDGE, at.size)
                assert np.array_equal(*f(x), equal_nan=True)
    finally:
        ctx.close()
