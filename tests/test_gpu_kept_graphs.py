"""A context's kept graphs through calls of other sizes, parameters and slots in between: solves and batches give, bit
for bit, what a fresh context gives, and contexts with every kind of graph close one after the other."""
import numpy as np
import pytest

import oracle as O
from rumb import _lib
from rumb.instances import mixture_instance

pytestmark = pytest.mark.gpu


def _solve(c, n, d, dt, kw):
    m, a, p = mixture_instance(n, d, K=10, N=100, seed=n)
    par = c.bm_params(O.beta_default(p.size), max_iter=150, abs_tol=1e-12, rel_tol=None, dtype=dt, **kw)
    r, fit, _ = c.bm_solve(c.bm_problem(n, m, a, p), par)
    return [r[k] for k in ("ub", "lb", "phi", "iters", "n_lb")], fit


def _batch(c, n, d, dt, kw, B, slots):
    m, a, p = mixture_instance(n, d, K=10, N=100, seed=n)
    P = np.clip(p[None, :] + np.random.default_rng(B).normal(0, 0.02, (B, p.size)), 0.0, 1.0)
    par = c.bm_params(O.beta_default(p.size), max_iter=100, abs_tol=1e-12, rel_tol=None, dtype=dt, **kw)
    res, _ = c.bm_solve_batch(c.bm_problem(n, m, a, p), par, P, slots=slots, want_fit=True)
    return [[r[k] for k in ("ub", "lb", "phi", "iters", "n_lb")] for r in res], np.stack([r["p_fit"] for r in res])


CALLS = [(_solve, 10, 0.5, "float64", {}), (_solve, 10, 0.3, "float64", {}), (_solve, 10, 0.5, "float32", dict(lb_every=2)),
         (_solve, 10, 0.5, "float32", {}), (_solve, 14, 0.02, "float32", dict(alpha=1.8)), (_solve, 14, 0.02, "float32", {}),
         (_solve, 13, 0.1, "mixed", dict(lb_every=2)), (_solve, 13, 0.1, "float64", dict(overlap_check=True)),
         (_solve, 6, 1.0, "float64", {}), (_solve, 7, 1.0, "float32", {}),
         (_batch, 10, 0.5, "float64", {}, 4, 4), (_batch, 10, 0.5, "float64", {}, 4, 2), (_batch, 10, 0.3, "float64", {}, 4, 4),
         (_batch, 10, 0.5, "float64", dict(alpha=1.8), 4, 4), (_batch, 13, 0.1, "float64", {}, 3, 2),
         (_batch, 12, 0.1, "float32", {}, 3, 3), (_batch, 12, 0.1, "float32", dict(lb_every=2), 3, 3)]


def test_calls_in_turn_equal_fresh_contexts():
    used = _lib.Context(0)
    want = []
    for f, *args in CALLS:
        c = _lib.Context(0)
        want.append(f(c, *args))
        c.close()
    for i in list(range(len(CALLS))) + list(range(len(CALLS)))[::-1] + [0, 10, 0, 11, 3, 2, 3]:
        f, *args = CALLS[i]
        got, fit = f(used, *args)
        assert got == want[i][0], CALLS[i][1:]
        np.testing.assert_array_equal(fit, want[i][1])
    used.close()
