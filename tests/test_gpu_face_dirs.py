"""The momentum kernels' face fluxes on grids that give a block one direction and on
one that gives it all three, with blocked cells scattered so that one-sided,
unassigned and carried-over derivatives occur everywhere: bit for bit against the
oracle."""
import types

import numpy as np
import pytest

from cases import MOM_DT, MOM_REN, momentum_inputs
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("central", [0, 1])
@pytest.mark.parametrize("cells", [(9, 12, 10), (20, 31, 24), (60, 52, 54)])
def test_calc_rhs_matches_oracle(cells, central):
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300.solver import PoissonContext
    P = W.make_problem(cells, (1.0, 1.0, 1.0), 1.0, True, (False,) * 3, [], nlevels=1)
    rng = np.random.default_rng(11)
    nv = P.nvert.copy()
    at = rng.choice(nv.size, nv.size // 8, replace=False)
    nv.ravel()[at] = rng.choice([0.05, 1.0, 3.0], at.size)
    P = types.SimpleNamespace(metrics=P.metrics, nvert=nv, ucont=P.ucont, bctype=P.bctype, semi=P.semi)
    L = O.OLevel(P.metrics[-1], nv, P.bctype, P.semi)
    ucat, p, uo, urm = momentum_inputs(nv.shape)
    ctx = PoissonContext().setup(P)
    try:
        r_g, u_g = ctx.calc_rhs(P.ucont, uo, urm, ucat, p, MOM_REN, MOM_DT, 5, 0, central=central)
        rc, r_o, u_o = O.calc_rhs(L, P.ucont, uo, urm, ucat, p, MOM_REN, MOM_DT, 5, 0, central)
        assert rc == 0
        assert np.ascontiguousarray(u_g).tobytes() == np.ascontiguousarray(u_o).tobytes()
        assert np.array_equal(r_g, r_o)
    finally:
        ctx.close()
