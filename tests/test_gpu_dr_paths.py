"""The two-kernel float64 iteration where a solve enters, leaves and shares it: batches whose slots stop and refill
out of step, kept states and warm starts, a mixed solve that hands over at its iteration limit, and the lattices
with one and two middle passes beyond the sizes the oracle reaches (n = 23, 24)."""
import numpy as np
import pytest

import oracle as O
from rumb import _lib
from rumb.instances import mixture_instance, rows_of, top_of_orders

pytestmark = pytest.mark.gpu


def _rows(n):
    return mixture_instance(n, min(0.2, 1500.0 / 2 ** n), K=8, N=100, seed=n)


@pytest.mark.parametrize("n", [13, 16, 19])
@pytest.mark.parametrize("warm", [False, True])
def test_batch_slots_refill_out_of_step(ctx, n, warm):
    """Five draws on two slots, three of them decided at their first check: the same kernels on the same values
    as a solve of its own, so the same bits."""
    m, a, p = _rows(n)
    P = np.clip(p[None, :] + np.random.default_rng(n).normal(0, 0.02, (5, p.size)), 0.0, 1.0)
    beta = O.beta_default(p.size)
    prob = ctx.bm_problem(n, m, a, p)
    kept = ctx.bm_solve(prob, ctx.bm_params(beta, max_iter=100, abs_tol=0.0, rel_tol=None), keep=True)[2] if warm else None
    below = np.array([1e6, np.nan, 1e6, np.nan, 1e6])
    par = ctx.bm_params(beta, max_iter=200, abs_tol=0.0, rel_tol=None, lb_every=2)
    res, info = ctx.bm_solve_batch(prob, par, P, below=below, warm=kept, slots=2, want_fit=True)
    assert info["slots"] == 2
    for b in range(5):
        one = ctx.bm_params(beta, max_iter=200, abs_tol=0.0, rel_tol=None, lb_every=2,
                            ub_target=None if np.isnan(below[b]) else below[b])
        r, fit, _ = ctx.bm_solve(ctx.bm_problem(n, m, a, P[b]), one, warm=kept)
        assert r["iters"] == (200 if np.isnan(below[b]) else 50)
        assert all(res[b][k] == r[k] for k in ("iters", "stop_reason", "ub", "lb", "phi", "n_lb"))
        np.testing.assert_array_equal(res[b]["p_fit"], fit)
    if kept:
        kept.close()


@pytest.mark.parametrize("n", [13, 16, 19, 21])
def test_kept_state_goes_on(ctx, n):
    """100 iterations kept and 100 more from there against 200 in one go: the state's way out and in rounds each
    value a few times, 1e-9 after 100 iterations as the other float64 tests."""
    m, a, p = _rows(n)
    beta = O.beta_default(p.size)
    prob = ctx.bm_problem(n, m, a, p)
    par = lambda it: ctx.bm_params(beta, max_iter=it, check=100, abs_tol=0.0, rel_tol=None)
    r0, _, kept = ctx.bm_solve(prob, par(100), keep=True)
    r1, _, _ = ctx.bm_solve(prob, par(100), warm=kept)
    kept.close()
    r2, _, _ = ctx.bm_solve(prob, par(200))
    for k, v in (("phi", r1["phi"]), ("ub", min(r0["ub"], r1["ub"])), ("lb", max(r0["lb"], r1["lb"]))):
        assert abs(v - r2[k]) <= 1e-9 * max(1.0, r2[k]), k


def test_mixed_solve_that_hands_over_at_its_limit(ctx):
    """The float32 leg stalls at the iteration limit: the kept state is its state, promoted."""
    n = 13
    m, a, p = _rows(n)
    beta = O.beta_default(p.size)
    prob = ctx.bm_problem(n, m, a, p)
    kw = dict(max_iter=100, abs_tol=0.0, rel_tol=None)
    rm, _, km = ctx.bm_solve(prob, ctx.bm_params(beta, dtype="mixed", stall_checks=1, stall_rtol=1.0, **kw), keep=True)
    assert rm["iters"] == rm["iters_f32"] == 100             # the second check is the limit
    r32, _, k32 = ctx.bm_solve(prob, ctx.bm_params(beta, dtype="float32", stall_checks=0, **kw), keep=True)
    assert r32["iters"] == 100
    go = ctx.bm_params(beta, max_iter=50, abs_tol=0.0, rel_tol=None)
    (x, fx, _), (y, fy, _) = ctx.bm_solve(prob, go, warm=km), ctx.bm_solve(prob, go, warm=k32)
    assert (x["ub"], x["lb"], x["phi"]) == (y["ub"], y["lb"], y["phi"])
    np.testing.assert_array_equal(fx, fy)
    km.close()
    k32.close()


@pytest.mark.parametrize("n", [21, 23, 24])
def test_middle_passes_against_the_transform_passes(ctx, monkeypatch, n):
    """Four iterations and a check against the transform passes with the prox (RUMB_FUSE pinned): n = 23 is the
    first with 9-bit tiles and a middle pass, n = 24 the first with two. 4 (n - 1) stages an iteration round
    differently: 1e-11 relative, as the iterate tests at a few iterations."""
    rng = np.random.default_rng(n)
    menus = np.unique(rng.integers(3, 1 << n, size=300))
    menus = menus[(menus & (menus - 1)) != 0]
    orders = np.stack([rng.permutation(n) for _ in range(8)])
    share = np.zeros((menus.size, n))
    np.add.at(share, (np.repeat(np.arange(menus.size), 8), top_of_orders(n, menus, orders).reshape(-1)), 0.125)
    m, a, p = rows_of(n, menus, share + 0.02 * rng.random(share.shape) * ((menus[:, None] >> np.arange(n)) & 1))
    prob = ctx.bm_problem(n, m, a, p)
    par = ctx.bm_params(O.beta_default(p.size), max_iter=4, check=4, abs_tol=0.0, rel_tol=None)
    got, fit, _ = ctx.bm_solve(prob, par)
    monkeypatch.setenv("RUMB_FUSE", "1")
    want, ref, _ = ctx.bm_solve(prob, par)
    for k in ("ub", "lb", "phi"):
        assert abs(got[k] - want[k]) <= 1e-11 * max(1.0, abs(want[k])), k
    np.testing.assert_allclose(fit, ref, rtol=0, atol=1e-11)
