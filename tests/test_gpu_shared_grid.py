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
