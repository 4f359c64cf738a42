"""Contexts of one grid in several threads: what the grid's contexts share and form on
first use (the face metric products, Contra2Cart's factors) is formed once, and the
results are those of the same calls one after another."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

THREADS = 4


def _contexts(P):
    from curvib_old_gb300.solver import PoissonContext
    donor = PoissonContext().setup(P)
    return [donor] + [PoissonContext().setup_like(donor, P.nvert) for _ in range(THREADS - 1)]


def test_first_projections_at_once():
    from curvib_old_gb300 import workload as W
    P = W.make_problem((24, 20, 28), (1.0, 1.0, 1.0), 1.0, True, (False,) * 3, [(0.5, 0.5, 0.5, 0.2)], nlevels=2)
    rng = np.random.default_rng(1)
    fields = [(rng.standard_normal(P.nvert.shape), rng.standard_normal(P.nvert.shape + (3,))) for _ in range(THREADS)]

    def calls(ctx, phi, u):
        return ctx.projection(phi, 1e-3, 1.0, u), ctx.contra2cart(u, np.zeros_like(u))

    one = _contexts(P)
    want = [calls(c, *f) for c, f in zip(one, fields)]
    size = one[0].geometry_bytes()[0]
    for c in one:
        c.close()
    for _ in range(8):
        ctxs = _contexts(P)
        got, errors, start = [None] * THREADS, [], threading.Barrier(THREADS)

        def work(q):
            try:
                start.wait()
                got[q] = calls(ctxs[q], *fields[q])
            except Exception as e:
                errors.append(e)

        threads = [threading.Thread(target=work, args=(q,)) for q in range(THREADS)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        try:
            assert not errors
            assert ctxs[0].geometry_bytes()[0] == size
            for g, w in zip(got, want):
                assert all(np.array_equal(a, b) for a, b in zip(g, w))
        finally:
            for c in ctxs:
                c.close()


def test_products_leave_nothing_behind_at_the_limit():
    """With not a byte left under the context's own limit, Projection's optional grid
    products are formed once or not at all: a second call takes no more memory."""
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300.solver import PoissonContext
    P = W.make_problem((24, 20, 28), (1.0, 1.0, 1.0), 1.0, True, (False,) * 3, [], nlevels=2)
    rng = np.random.default_rng(2)
    phi, u = rng.standard_normal(P.nvert.shape), rng.standard_normal(P.nvert.shape + (3,))
    free, full = PoissonContext().setup(P), PoissonContext().setup(P)
    try:
        want = free.projection(phi, 1e-3, 1.0, u)
        size, limit = full.geometry_bytes()[0], full.device_bytes()
        assert limit >= size + 72 * P.nvert.size  # the products themselves fit
        full.set_device_limit(limit)
        sizes = []
        for _ in range(3):
            assert np.array_equal(full.projection(phi, 1e-3, 1.0, u), want)
            sizes.append(full.geometry_bytes()[0] - size)
        assert sizes[0] in (0, 72 * P.nvert.size) and sizes[1:] == [sizes[0]] * 2
    finally:
        free.close()
        full.close()


@pytest.mark.parametrize("first", ["contra2cart", "projection"])
def test_contra2cart_fits_with_its_factors_alone(first):
    """A limit that leaves room for Contra2Cart's factors (80 bytes a cell) and nothing
    else on the grid: the arrays that its kernel and Projection's can do without stay
    away, whichever call comes first, and the results are the same."""
    from curvib_old_gb300 import workload as W
    from curvib_old_gb300.solver import PoissonContext
    P = W.make_problem((24, 20, 28), (1.0, 1.0, 1.0), 1.0, True, (False,) * 3, [], nlevels=1)
    rng = np.random.default_rng(3)
    phi, u = rng.standard_normal(P.nvert.shape), rng.standard_normal(P.nvert.shape + (3,))
    free, full = PoissonContext().setup(P), PoissonContext().setup(P)
    try:
        n = P.nvert.size
        want = free.projection(phi, 1e-3, 1.0, u), free.contra2cart(u, np.zeros_like(u))
        limit = full.geometry_bytes()[0] + 80 * n
        assert limit >= full.device_bytes() + 48 * n  # the context's own part of the call
        full.set_device_limit(limit)
        if first == "projection":
            assert np.array_equal(full.projection(phi, 1e-3, 1.0, u), want[0])
        assert np.array_equal(full.contra2cart(u, np.zeros_like(u)), want[1])
        assert np.array_equal(full.projection(phi, 1e-3, 1.0, u), want[0])
        assert full.geometry_bytes()[0] == limit
    finally:
        free.close()
        full.close()
