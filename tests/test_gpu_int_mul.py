"""The momentum kernels' integer-pipe products at the edges of their range:
values beside it, beyond it and not finite among ordinary ones (those faces
take the FP64 multiplies), and grids whose metrics are beyond it (all of them
do).  Bit for bit against the CPU oracle, a NaN equal to a NaN."""
import types

import numpy as np
import pytest

from cases import MOM_DT, MOM_REN, build, momentum_inputs
from oracle import oracle as O

pytestmark = pytest.mark.gpu
EDGE = [0.0, -0.0, 2.0**-510, 2.0**-511, -(2.0**-512), 2.0**-700, 5e-324, 2.0**511, 2.0**512, -(2.0**600), 1e308,
        np.inf, -np.inf, np.nan]


def _same(a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    nan = np.isnan(a)
    return np.array_equal(nan, np.isnan(b)) and a[~nan].tobytes() == b[~nan].tobytes()


@pytest.mark.parametrize("grid", ["plain", "small_metrics", "large_metrics"])
@pytest.mark.parametrize("values", ["plain", "edge"])
def test_products_match_oracle(grid, values):
    from curvib_old_gb300.solver import PoissonContext
    c = build("box_sphere")
    metrics = [dict(m) for m in c["metrics"]]
    if grid != "plain":
        f = 2.0 ** (-300 if grid == "small_metrics" else 300)
        for nm in ("JCsi", "JEta", "JZet"):
            metrics[-1][nm] = metrics[-1][nm] * f
    ucat, p, uo, urm = momentum_inputs(c["nvert"].shape)
    uc = c["ucont"].copy()
    if values == "edge":
        rng = np.random.default_rng(5)
        for a in (ucat, uc):
            at = rng.choice(a.size, a.size // 40, replace=False)
            a.ravel()[at] = rng.choice(EDGE, at.size)
    P = types.SimpleNamespace(metrics=metrics, nvert=c["nvert"], ucont=uc, bctype=c["bctype"], semi=c["semi"])
    ctx = PoissonContext().setup(P)
    try:
        L = O.OLevel(metrics[-1], c["nvert"], c["bctype"], c["semi"])
        with np.errstate(all="ignore"):
            assert _same(ctx.viscous(ucat, MOM_REN), O.viscous(L, ucat, MOM_REN))
            r_g, u_g = ctx.calc_rhs(uc, uo, urm, ucat, p, MOM_REN, MOM_DT, 5, 0)
            rc, r_o, u_o = O.calc_rhs(L, uc, uo, urm, ucat, p, MOM_REN, MOM_DT, 5, 0)
        assert rc == 0 and _same(u_g, u_o) and _same(r_g, r_o)
    finally:
        ctx.close()


@pytest.mark.parametrize("values", ["plain", "edge"])
@pytest.mark.parametrize("dt,st", [(1e-3, 1.0), (0.7, 0.3), (2.0**-520, 1.0), (1e-3, 2.0**515)])
@pytest.mark.parametrize("name", ["box_sphere", "triply_periodic"])
def test_projection_and_rhs_match_oracle(name, dt, st, values):
    """PoissonRHS and Projection with ordinary and extreme time factors; the
    fluxes and pressures ordinary or with values beside and beyond the range."""
    from curvib_old_gb300.solver import PoissonContext
    c = build(name)
    rng = np.random.default_rng(7)
    uc, phi = c["ucont"].copy(), rng.standard_normal(c["nvert"].shape)
    if values == "edge":
        for a in (phi, uc):
            at = rng.choice(a.size, a.size // 40, replace=False)
            a.ravel()[at] = rng.choice(EDGE, at.size)
    P = types.SimpleNamespace(metrics=c["metrics"], nvert=c["nvert"], ucont=uc, bctype=c["bctype"], semi=c["semi"])
    ctx = PoissonContext().setup(P)
    try:
        L = O.OLevel(c["metrics"][-1], c["nvert"], c["bctype"], c["semi"])
        with np.errstate(all="ignore"):
            b_o, _ = O.poisson_rhs(L, uc, dt, st)
            b_g, _ = ctx.poisson_rhs(uc, dt, st)
            _, phi_o, uc_o = O.update_and_project(L, np.zeros_like(phi), phi, uc, dt, st)
            _, phi_g = ctx.update_pressure(np.zeros_like(phi), phi)
            uc_g = ctx.projection(phi_g, dt, st, uc)
        assert _same(b_g, b_o) and _same(phi_g, phi_o) and _same(uc_g, uc_o)
    finally:
        ctx.close()
