"""The iteration's sequence (transform windows, prox form, fused passes) follows from n and the state type:
a float32 state's fit depends on it by 0.1-1 %, so fresh contexts, batches and contexts with other solves
behind them give the same bits."""
import numpy as np
import pytest

import oracle as O
from rumb import _lib
from rumb.instances import mixture_instance

pytestmark = pytest.mark.gpu


def _rows(n):
    return mixture_instance(n, 0.3 if n <= 10 else min(0.1, 1500.0 / 2 ** n), K=8, N=100, seed=n)


def _bits(r, fit):
    return (r["ub"], r["lb"], r["phi"], r["iters"], fit.tobytes())


@pytest.mark.parametrize("n", range(8, 23))
@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_fresh_contexts_and_batches_agree(n, dtype):
    m, a, p = _rows(n)
    par = _lib.Context.bm_params(O.beta_default(p.size), max_iter=100 if n <= 18 else 50, abs_tol=0.0, rel_tol=None, dtype=dtype)
    got = []
    for _ in range(4 if n <= 18 else 2):
        c = _lib.Context(0)
        got.append(_bits(*c.bm_solve(c.bm_problem(n, m, a, p), par)[:2]))
        c.close()
    c = _lib.Context(0)                                    # a batch with no solve before it
    res, _ = c.bm_solve_batch(c.bm_problem(n, m, a, p), par, p[None, :], want_fit=True)
    got.append(_bits(res[0], res[0]["p_fit"]))
    it = c.bm_iterate(c.bm_problem(n, m, a, p), par, None, 5, cold_start=True)
    c.close()
    assert all(g == got[0] for g in got)
    c = _lib.Context(0)                                    # iterates with and without a solve before them
    c.bm_solve(c.bm_problem(n, m, a, p), par)
    again = c.bm_iterate(c.bm_problem(n, m, a, p), par, None, 5, cold_start=True)
    c.close()
    for k in ("x2", "s", "y", "z"):
        np.testing.assert_array_equal(it[k], again[k])


@pytest.mark.parametrize("n,form", [(8, 2), (12, 4), (15, 3), (17, 0), (18, 0), (19, 6), (20, 6), (21, 6), (22, 6), (23, 0)])
def test_float32_member_sums_keep_their_order(ctx, monkeypatch, n, form):
    """The order of a menu's sums at each n: the one of the tile and lanes forms up to n = 18 and from n = 23,
    the two-array tile's between (pinned here to another form of the same order)."""
    m, a, p = _rows(n)
    par = ctx.bm_params(O.beta_default(p.size), max_iter=100 if n <= 18 else 50, abs_tol=0.0, rel_tol=None, dtype="float32")
    got = _bits(*ctx.bm_solve(ctx.bm_problem(n, m, a, p), par)[:2])
    monkeypatch.setenv("RUMB_PROX_FORM", str(form))
    c = _lib.Context(0)
    assert _bits(*c.bm_solve(c.bm_problem(n, m, a, p), par)[:2]) == got
    c.close()
