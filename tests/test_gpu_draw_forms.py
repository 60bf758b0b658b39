"""The screen kernel's forms (csrc/draws.cu): four and two draws a CTA with a ragged last CTA, from all draws and from
a list of them, and one draw a CTA with seen kept by menu or summed again for every row, by size and by how many
CTAs an SM holds. Whole weights and counts: the sums are exact in any order, so every row is bit for bit numpy's."""
from types import SimpleNamespace

import numpy as np
import pytest

from rumb import _lib
from rumb import bootstrap as BS
from rumb.instances import panel_instance

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [591, 592, 593, 1183, 1184, 1187])
def test_draws_sharing_a_cta_match_host(ctx, B):
    panel, (m, a, p) = panel_instance(10, 0.3, 80, 8, 5, seed=7)
    d = BS.Draws(panel, m, a, p, B=B, weights="multinomial", seed=3)
    g = _lib.DrawRows(ctx, d.W, d.lists, d.p_hat)
    r_n, eps_n, _ = BS.scaling(d.R)
    host = d.rows(np.arange(B))
    idx = np.random.default_rng(B).permutation(B)
    np.testing.assert_array_equal(g.rows(idx), host[idx])
    P = BS.perturb(d.p_hat, host, r_n, eps_n)
    np.testing.assert_array_equal(g.rows(np.arange(B), eps_n * r_n), P)
    fit = np.clip(d.p_hat + 0.01 * np.sin(np.arange(d.M)), 0.0, 1.0)
    dev, ub = g.screen(fit, eps_n * r_n)
    np.testing.assert_allclose(dev, np.linalg.norm(host - d.p_hat, axis=1), rtol=1e-12, atol=0)
    np.testing.assert_allclose(ub, np.linalg.norm(P - fit, axis=1), rtol=1e-12, atol=0)
    g.close()


@pytest.mark.parametrize("k", [3, 4])
@pytest.mark.parametrize("R,U,B", [(300, 26000, 40), (300, 25300, 149), (300, 25300, 40), (1000, 15000, 149), (1000, 15000, 148),
                                   (12000, 3000, 149), (7000, 6000, 149), (20000, 5000, 20), (20480, 100, 20)])
def test_one_draw_a_cta_with_and_without_seen_kept(ctx, R, U, B, k):
    rng = np.random.default_rng(U)
    resp = np.repeat(np.arange(R), 20)
    at = rng.integers(0, U, resp.size)                       # the offers' menus; some menus are offered to nobody
    rows = np.repeat(np.arange(U), k)
    ch = k * at + rng.integers(0, k, at.size)
    o, c = np.argsort(at, kind="stable"), np.argsort(ch, kind="stable")
    ptr = lambda v, n: np.concatenate([[0], np.cumsum(np.bincount(v, minlength=n))])
    cnt = rng.integers(1, 4, at.size).astype(float)
    lists = SimpleNamespace(menu_ptr=ptr(at, U), menu_resp=resp[o], menu_cnt=cnt[o], row_ptr=ptr(ch, k * U), row_resp=resp[c],
                            row_cnt=cnt[c], row_menu=rows)
    W = rng.integers(0, 3, (B, R)).astype(float)
    p_hat = rng.random(k * U)
    g = _lib.DrawRows(ctx, W, lists, p_hat)
    got = g.rows(np.arange(B))
    dev, _ = g.screen(None, 0.5)
    want = np.empty((B, k * U))
    for b in range(B):
        seen = np.bincount(at, weights=W[b, resp] * cnt, minlength=U)[rows]
        chose = np.bincount(ch, weights=W[b, resp] * cnt, minlength=k * U)
        want[b] = np.where(seen > 0, chose / np.where(seen > 0, seen, 1.0), p_hat)
    np.testing.assert_array_equal(got, want)
    np.testing.assert_allclose(dev, np.linalg.norm(want - p_hat, axis=1), rtol=1e-12, atol=0)
    g.close()
