"""What a batch leaves with its context to save the next one's allocations (certificate slots, uploaded draws) is given
back when a later call is short of memory, so that a solve fits where its plan says it does."""
import numpy as np
import pytest
import torch

import oracle as O
from rumb import _lib
from rumb.instances import mixture_instance

pytestmark = pytest.mark.gpu


def test_solve_fits_beside_what_a_batch_left():
    c = _lib.Context(0)
    m, a, p = mixture_instance(16, 0.02, K=8, N=100, seed=1)
    P = np.clip(p[None, :] + np.random.default_rng(1).normal(0, 0.02, (24, p.size)), 0.0, 1.0)
    prob = c.bm_problem(16, m, a, p)
    par = c.bm_params(O.beta_default(p.size), max_iter=50, abs_tol=0.0, rel_tol=None)
    first, info = c.bm_solve_batch(prob, par, P, slots=24, want_fit=True)
    assert info["slots"] == 24
    m2, a2, p2 = mixture_instance(18, 0.005, K=8, N=100, seed=2)
    go = c.bm_params(O.beta_default(p2.size), max_iter=50, abs_tol=0.0, rel_tol=None)
    # the batch leaves 24 slots of 10 MB; a solve of n = 18 takes 230 MB, 44 of them certificate arrays. With 130 MB
    # free it fits only if the slots go back.
    need = _lib.bm_plan(18, p2.size, "float64")
    spare = c.mem_info()[0] - torch.cuda.mem_get_info()[0]
    assert (200 << 20) <= spare <= (384 << 20)               # counted as free for this context
    fill = torch.empty(torch.cuda.mem_get_info()[0] - need + (100 << 20), dtype=torch.uint8, device="cuda")
    try:
        got, fit, _ = c.bm_solve(c.bm_problem(18, m2, a2, p2), go)
    finally:
        del fill
        torch.cuda.empty_cache()
    fresh = _lib.Context(0)
    want, ref, _ = fresh.bm_solve(fresh.bm_problem(18, m2, a2, p2), go)
    fresh.close()
    assert (got["ub"], got["lb"]) == (want["ub"], want["lb"])
    np.testing.assert_array_equal(fit, ref)
    again, info = c.bm_solve_batch(prob, par, P, slots=24, want_fit=True)      # and a batch after it
    for x, y in zip(first, again):
        assert (x["ub"], x["lb"], x["iters"]) == (y["ub"], y["lb"], y["iters"])
        np.testing.assert_array_equal(x["p_fit"], y["p_fit"])
    c.close()


def test_batch_takes_what_the_other_state_dtype_left():
    """A float32 batch leaves 60 MB of draws; with 40 MB free a float64 batch's own draws fit only in their place."""
    c = _lib.Context(0)
    m, a, p = mixture_instance(10, 1.0, K=8, N=100, seed=1)
    B = (60 << 20) // (8 * p.size)
    P = np.clip(p[None, :] + np.random.default_rng(1).normal(0, 0.02, (B, p.size)), 0.0, 1.0)
    prob = c.bm_problem(10, m, a, p)
    run = lambda dt: c.bm_solve_batch(prob, c.bm_params(O.beta_default(p.size), max_iter=50, abs_tol=0.0, rel_tol=None, dtype=dt),
                                      P, below=np.full(B, 1e6), slots=1)[0]
    run("float32")
    c.bm_solve(prob, c.bm_params(O.beta_default(p.size), max_iter=50, abs_tol=0.0, rel_tol=None))
    fill = torch.empty(torch.cuda.mem_get_info()[0] - (40 << 20), dtype=torch.uint8, device="cuda")
    try:
        got = run("float64")
    finally:
        del fill
        torch.cuda.empty_cache()
    want = run("float64")
    assert [(r["ub"], r["lb"], r["iters"]) for r in got] == [(r["ub"], r["lb"], r["iters"]) for r in want]
    c.close()
