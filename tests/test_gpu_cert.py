"""The certificate's kernels at the edges of their launch shapes: the largest lattice of the
one-CTA recursions and the smallest of the layer launches (n = 12, 13), few rows and more rows than
one round of the row sums' loads (8 x 1024), and a batch's slots checked together with a lower bound
every second check only."""
import numpy as np
import pytest

import oracle as O
from rumb.instances import config_instance, mixture_instance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,rows", [(2, None), (11, 1), (12, 1023), (12, 8193), (13, 1025), (13, 17000)])
def test_push_and_lower_bound_at_the_edges(ctx, n, rows):
    menu, alt, p = mixture_instance(n, 1.0, K=5, N=100, seed=n)
    if rows is not None:
        keep = np.sort(np.random.default_rng(rows).choice(menu.size, rows, replace=False))
        menu, alt, p = menu[keep], alt[keep], p[keep]
    obs = O.slab_index(n, menu, alt)
    x = np.random.default_rng(n).random(n << (n - 1)) * 0.3
    ub_ref, xub = O.push_ub64(n, x, obs, p)
    ub, fit = ctx.push_ub64(n, x, menu, alt, p)
    # the tolerances of test_push_and_lower_bound_match_oracle: float64 sums of these many rows
    assert abs(ub - ub_ref) <= 1e-11 * max(1.0, ub_ref)
    np.testing.assert_allclose(fit, xub[obs], rtol=0, atol=1e-12)
    lb_ref = O.fw_lb64(n, obs, x[obs], p)
    assert abs(ctx.fw_lb64(n, menu, alt, x[obs], p) - lb_ref) <= 1e-10 * max(1.0, lb_ref)


def test_batch_lower_bound_every_second_check(ctx):
    n, m, a, p = config_instance("n10_all_k20")
    P = np.clip(p[None, :] + np.random.default_rng(1).normal(0, 0.02, (5, p.size)), 0.0, 1.0)
    par = ctx.bm_params(O.beta_default(p.size), abs_tol=5e-4, rel_tol=None, dtype="float64", lb_every=2)
    res, info = ctx.bm_solve_batch(ctx.bm_problem(n, m, a, p), par, P, slots=2, want_fit=True)
    assert info["slots"] == 2                               # refilled slots: their checks fall out of step
    for b in range(P.shape[0]):
        one, fit, _ = ctx.bm_solve(ctx.bm_problem(n, m, a, P[b]), par)
        assert res[b]["iters"] == one["iters"] and res[b]["n_lb"] == one["n_lb"]
        assert abs(res[b]["ub"] - one["ub"]) <= 1e-12 and abs(res[b]["lb"] - one["lb"]) <= 1e-12
        np.testing.assert_allclose(res[b]["p_fit"], fit, rtol=0, atol=1e-12)
