"""The set-up's operators at the edges of its integer products and of its shortcut
for open cells: metrics beyond the products' range (those rows take the FP64
multiplies), zero metrics, and nvert values of either sign of zero, below, at and
above 0.1.  The 19 weights equal the oracle's matrix bit for bit, and the FP32 rows
follow them."""
import types

import numpy as np
import pytest

from oracle import oracle as O
from parity_util import weights_to_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 2.0**-300, 2.0**300, 0.0])
@pytest.mark.parametrize("cells,per", [((10, 12, 8), (0, 0, 0)), ((12, 36, 8), (1, 0, 1))])
def test_weights_match_oracle(cells, per, scale):
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300.solver import PoissonContext
    P = W.make_problem(cells, (1.0, 1.0, 1.0), 1.0, True, tuple(map(bool, per)), [], nlevels=2)
    m = dict(P.metrics[1])
    for nm in ("JCsi", "JEta", "JZet"):
        m[nm] = m[nm] * scale
    nv = P.nvert.copy()
    rng = np.random.default_rng(4)
    inner = nv[1:-1, 1:-1, 1:-1]
    at = rng.choice(inner.size, inner.size // 9, replace=False)
    v = inner.ravel()
    v[at] = rng.choice([-0.0, 5e-324, 0.05, 0.1, np.nextafter(0.1, 1.0), 1.0, 3.0], at.size)
    nv[1:-1, 1:-1, 1:-1] = v.reshape(inner.shape)
    P = types.SimpleNamespace(metrics=[P.metrics[0], m], nvert=nv, ucont=P.ucont, bctype=P.bctype, semi=P.semi)
    L = O.OLevel(m, nv, P.bctype, P.semi)
    ctx = PoissonContext().setup(P)
    try:
        A = O.lhs_csr(L)
        d = A - weights_to_csr(ctx.weights(1), ctx.shapes[1], P.bctype)
        assert d.nnz == 0 or np.abs(d.data).max() == 0.0
        if scale == 1.0:
            x = rng.standard_normal(ctx.shapes[1]).astype(np.float32)
            y = (A @ x.astype(np.float64).ravel()).reshape(x.shape)
            assert np.abs(ctx.apply_f32(1, x) - y).max() <= 2e-6 * abs(A).max() * np.abs(x).max() * 4
    finally:
        ctx.close()
