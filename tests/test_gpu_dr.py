"""The two-kernel float64 iteration (csrc/dr.cu) against the oracle at every window shape: one and two
high-window exchanges (n = 13..20), middle passes (n = 21, 22), both p_hat lane groups (n <= 16 and
above), menus without, with some and with all members observed, and start states that no iteration
leaves behind (s and y both positive, x2 off the simplex)."""
import numpy as np
import pytest

import oracle as O
from rumb.instances import mixture_instance

pytestmark = pytest.mark.gpu


def _rows(n):
    """Rows of a sparse design, one row in five left out: menus observed in full and in part."""
    m, a, p = mixture_instance(n, min(0.2, 400.0 / 2 ** n), K=8, N=100, seed=n)
    keep = np.random.default_rng(n).random(m.size) > 0.2
    return m[keep], a[keep], p[keep]


@pytest.mark.parametrize("n", [13, 14, 15, 16, 17, 18, 19, 20, 21, 22])
def test_two_kernel_iteration_tracks_oracle(ctx, n):
    menu, alt, p = _rows(n)
    O.set_threads(0)
    bm = O.BMOracle(n, menu, alt, p)
    prob, par = ctx.bm_problem(n, menu, alt, p), ctx.bm_params(O.beta_default(p.size))
    rng = np.random.default_rng(100 + n)
    m2 = n << (n - 1)
    free = {k: rng.random(m2) * s for k, s in (("x2", 0.5), ("s", 0.1), ("y", 0.1), ("z", 0.1))}
    for start, iters in ((None, 3), (free, 2)):
        if start is not None:
            bm.set_state({k: v.copy() for k, v in start.items()})
        st = ctx.bm_iterate(prob, par, start, iters, cold_start=start is None)
        bm.iterate(iters)
        # 4 (n - 1) butterfly stages an iteration round differently: 1e-11 of the largest value, as
        # the other iterate tests at a few iterations
        for name in ("x2", "s", "y", "z"):
            ref = getattr(bm, name)
            d = np.max(np.abs(st[name] - ref))
            assert d <= 1e-11 * max(1.0, float(np.max(np.abs(ref)))), (name, start is None, d)
