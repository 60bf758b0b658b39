"""Launching ahead changes when kernels are scheduled, never what they compute, where kernels really go ahead: the
iteration up to n = 10 in graphs and at every n launched one by one, and the pricing layers, whose sums are formed
before the wait, with lists and without, on designs with layers of a warp per alternative, with other scores in each
of several calls in a row. Child processes with RUMB_PDL=1 and 0 (read once per process) give the same bits."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

_WORK = r'''
import os, sys
import numpy as np
sys.path[:0] = [%(pkg)r, %(oracle)r]
from rumb import _lib
from rumb.instances import mixture_instance
import oracle as O
ctx = _lib.Context(0)
out = {}
for n in (8, 9, 10, 12, 14):
    m, a, p = mixture_instance(n, 0.3 if n <= 10 else 0.05, K=8, N=200, seed=n)
    for dt in ("float64", "float32"):
        for graph in (True, False):
            par = ctx.bm_params(O.beta_default(p.size), max_iter=100, abs_tol=0.0, rel_tol=None, dtype=dt, use_graph=graph)
            r, fit, _ = ctx.bm_solve(ctx.bm_problem(n, m, a, p), par)
            out["%%d_%%s_%%d" %% (n, dt, graph)] = np.concatenate([[r["ub"], r["lb"], r["phi"]], fit])
os.environ["RUMB_MASK_FORM"] = os.environ["RUMB_STREAM_FORM"] = "layer"
for n, density in ((9, 0.5), (13, 0.05), (17, 0.002)):
    m, a, p = mixture_instance(n, density, K=8, N=100, seed=n)
    menus, _, p32, offsets, _ = O.cg_layout(n, m, a, p)
    rng = np.random.default_rng(n)
    scores = [rng.normal(0, 0.1, p32.size).astype(np.float32) for _ in range(4)]
    for mode in ("mask", "f32", "u16", "u24"):
        for lists in (True, False):
            pr = _lib.Pricer(ctx, n, menus, offsets, mode=mode, lists=lists, stream=mode == "f32")
            for i in range(12):
                v, r, mg = pr.price(scores[i %% 4])
                out["%%d_%%s_%%d_%%d" %% (n, mode, lists, i)] = np.concatenate([[v, mg], r])
            pr.close()
np.savez(sys.argv[1], **out)
'''


def _run(path, pdl):
    code = _WORK % dict(pkg=os.path.join(ROOT, "rum-testing-gpu_b200"), oracle=os.path.join(ROOT, "oracle"))
    r = subprocess.run([sys.executable, "-c", code, path], env=dict(os.environ, RUMB_PDL=pdl), capture_output=True, text=True,
                       timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    return np.load(path)


def test_launching_ahead_gives_the_same_bits(tmp_path):
    on, off = _run(str(tmp_path / "on.npz"), "1"), _run(str(tmp_path / "off.npz"), "0")
    assert set(on.files) == set(off.files)
    for k in on.files:
        np.testing.assert_array_equal(on[k], off[k], err_msg=k)
        if k.count("_") == 3:                                # the same scores again: the same answer
            n, mode, lists, i = k.rsplit("_", 3)
            np.testing.assert_array_equal(on[k], on["%s_%s_%s_%d" % (n, mode, lists, int(i) % 4)], err_msg=k)
