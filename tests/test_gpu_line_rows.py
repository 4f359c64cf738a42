"""The rows of the FP64 line relaxation (80 bytes a cell of a level that takes it) are
optional: only FP64 zebra solves form them, a context that fits without them sets up
and solves, and they make way for what a call cannot do without.  A solve without them
is the tile kernels', equal up to rounding (tests/test_gpu_lines.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CELLS = (64, 16, 304)
N = 66 * 18 * 306  # mx even: as many slots in the colour-split rows as cells


@pytest.fixture(scope="module")
def case():
    from curvib_old_gb300 import _lib
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300.solver import PoissonContext
    P = W.make_problem(CELLS, (1.0, 1.0, 1.0), 1.0, False, (False,) * 3, [(0.5, 0.5, 0.5, 0.2)], nlevels=4)
    ctx = PoissonContext().setup(P)
    c = {"P": P, "setup": ctx.device_bytes()}
    uc, _, _ = ctx.volume_flux_rev(P.ucont)
    c["u"] = uc
    c["b"], _ = ctx.poisson_rhs(uc, 1e-3, 1.0)
    ctx.solve(c["b"], precision=_lib.MIXED, rtol=1e-8)
    c["mixed"] = ctx.device_bytes()
    c["phi"], c["st"] = ctx.solve(c["b"], precision=_lib.FP64, rtol=1e-8)
    c["fp64"] = ctx.device_bytes()
    assert _choice(ctx) == "lines"
    yield c
    ctx.close()


def _choice(ctx):
    return ctx.tuning()["line_sweep"][-1]["zebra_f64"]["choice"]


def _same(c, phi, st):
    assert st["iterations"] == c["st"]["iterations"]
    assert np.linalg.norm(phi - c["phi"]) <= 1e-10 * np.linalg.norm(c["phi"])


def test_only_fp64_solves_hold_them(case):
    assert case["fp64"] == case["mixed"] + 80 * N


def test_setup_and_solve_where_the_rest_fits(case):
    """The limit leaves the set-up what it takes at its fullest, the nine FP64
    coefficients a cell beside its arrays, which is less than the rows."""
    from curvib_old_gb300 import _lib
    from curvib_old_gb300.solver import PoissonContext
    ctx = PoissonContext()
    try:
        ctx.set_device_limit(case["setup"] + 72 * N)
        ctx.setup(case["P"])
        assert ctx.device_bytes() == case["setup"]
        ctx.set_device_limit(case["mixed"])
        for _ in range(3):  # as launched, captured, replayed
            _same(case, *ctx.solve(case["b"], precision=_lib.FP64, rtol=1e-8))
        assert _choice(ctx) != "lines" and ctx.device_bytes() <= case["mixed"]
        # with room again, the next set-up takes them
        ctx.set_device_limit(0)
        ctx.set_nvert(case["P"].nvert)
        for _ in range(3):
            phi, st = ctx.solve(case["b"], precision=_lib.FP64, rtol=1e-8)
        assert _choice(ctx) == "lines" and np.array_equal(phi, case["phi"]) and st["iterations"] == case["st"]["iterations"]
    finally:
        ctx.close()


def test_they_make_way(case):
    from curvib_old_gb300 import _lib
    from curvib_old_gb300.solver import PoissonContext
    ctx = PoissonContext().setup(case["P"])
    try:
        want = ctx.solve(case["b"], precision=_lib.FP64, rtol=1e-8)
        before = ctx.device_bytes()
        ctx.set_device_limit(before + 48 * N - 8)  # Contra2Cart's two fields but eight bytes
        u = ctx.contra2cart(case["u"], np.zeros_like(case["u"]))
        assert ctx.device_bytes() == before + (48 - 80) * N and _choice(ctx) != "lines"
        for _ in range(3):
            _same(case, *ctx.solve(case["b"], precision=_lib.FP64, rtol=1e-8))
        ctx.set_device_limit(0)
        assert np.array_equal(u, ctx.contra2cart(case["u"], np.zeros_like(case["u"])))
        assert np.array_equal(want[0], case["phi"])
    finally:
        ctx.close()
