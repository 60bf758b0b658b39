"""The measured cases: the calls a program makes of this library, over the sizes it makes them at.

    listed()            the cases, each a dict of plain values with its name
    draw(rng)           one more case of the same ranges
    prepare(case, seed) what the program holds before the call (data, contexts, plans, weights)
    run(state)          one call through the public entry points, and its outputs
    work(case)          bytes and operations the call cannot do without
    exact(case, seed)   the same outputs in 64 bits by plain torch / numpy

Kinds: "solve" a certified BM-ADMM distance of a fixed iteration budget (RUM.session().solve; the
smallest one is RUM.calculate_distance at its default tolerances); "batch" a chunk of bootstrap
draws solved together from p_hat's kept state; "price" one Flow-CG pricing call; "flow_cg" a whole
column-generation call; "screen" the bootstrap's screen of all draws; "mlp" the learned warm
start's loss and gradient.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rum-testing-gpu_b200"))

from rumb import RUM, _lib, bootstrap, flow_cg  # noqa: E402
from rumb.instances import panel_instance, rows_of, top_of_orders  # noqa: E402
from rumb.rum_solver import context  # noqa: E402

ALPHA, P_COND = 1.95, math.sqrt(2.0)          # bm_admm's defaults
DT = {"float64": torch.float64, "float32": torch.float32}


def listed():
    return [
        # the smallest call: a survey of 8 alternatives, every menu asked, default tolerances
        dict(name="distance_n8_all_menus", kind="solve", n=8, density=1.0, dtype="float64", iters=2000, tol=True),
        # an ordinary laboratory design with an odd number of alternatives, a tenth of the menus
        dict(name="solve_n13_f64", kind="solve", n=13, density=0.1, dtype="float64", iters=600, tol=False),
        # the benchmark's workload: 18 alternatives, 1 % of the menus; the certified solve is 43,850
        # such iterations with a check every 50
        dict(name="solve_n18_f64", kind="solve", n=18, density=0.01, dtype="float64", iters=200, tol=False),
        # its first leg in mixed precision: the float32 state
        dict(name="solve_n18_f32", kind="solve", n=18, density=0.01, dtype="float32", iters=200, tol=False),
        # the paper-sized instance
        dict(name="solve_n20_f64", kind="solve", n=20, density=0.01, dtype="float64", iters=200, tol=False),
        # the largest lattice that is iterated in earnest, few menus asked
        dict(name="solve_n22_f64", kind="solve", n=22, density=0.001, dtype="float64", iters=100, tol=False),
        # bootstrap: one chunk of draws from p_hat's kept state (12 alternatives, a panel)
        dict(name="batch_n12_24draws", kind="batch", n=12, density=0.1, dtype="float64", draws=24, iters=200),
        # bootstrap screen: every draw's two norms over a panel's rows
        dict(name="screen_n16_2000draws", kind="screen", n=16, density=0.02, respondents=520, draws=2000),
        # Flow-CG pricing: the sweep of one column at the sparse n = 18 design, the default storage
        # where the lattice is large
        dict(name="price_n18_u24", kind="price", n=18, menus="density", density=0.005, mode="u24"),
        # pricing at large n from binary menus, storage by mask
        dict(name="price_n26_pairs_mask", kind="price", n=26, menus="pairs", density=0.0, mode="mask"),
        # a whole Flow-CG call: columns until its tolerances or the column limit
        dict(name="flow_cg_n14", kind="flow_cg", n=14, density=0.01, columns=100),
        # the learned warm start's training step: loss and gradient of one batch of solved draws
        dict(name="mlp_301_1024", kind="mlp", width_in=301, hidden=1024, rows=1024),
    ]


def draw(rng):
    kind = rng.choice(["solve"] * 6 + ["batch", "price", "price", "flow_cg", "screen", "mlp"])
    if kind == "solve":
        n = rng.randint(8, 22)
        # the pushed point of an early iterate of a large lattice sits on entries that are zero up to rounding, so
        # the budgets stay where its values are settled to the accuracy they are compared at
        iters = 50 * (rng.randint(6, 12) if n <= 15 else rng.randint(2, 4) if n <= 20 else rng.randint(1, 2))
        lo, hi = (0.3, 1.0) if n <= 10 else (0.03, 0.2) if n <= 13 else (0.01, 0.05) if n <= 16 else (0.003, 0.012)
        if n >= 20:
            lo, hi = 0.0008, 0.003
        return dict(kind="solve", n=n, density=round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 5),
                    dtype=rng.choice(["float64", "float64", "float64", "float32"]), iters=iters, tol=False)
    if kind == "batch":
        n = rng.randint(9, 15)
        return dict(kind="batch", n=n, density=round(rng.uniform(0.03, 0.3) if n <= 12 else rng.uniform(0.01, 0.05), 4),
                    dtype="float64", draws=rng.randint(3, 32 if n <= 13 else 10), iters=50 * rng.randint(2, 5))
    if kind == "price":
        if rng.random() < 0.5:
            return dict(kind="price", n=rng.randint(10, 18), menus="density", density=round(rng.uniform(0.002, 0.01), 5),
                        mode=rng.choice(["mask", "f32", "u16", "u24"]))
        return dict(kind="price", n=rng.randint(16, 26), menus="pairs", density=0.0,
                    mode=rng.choice(["mask", "f32", "u16", "u24"]))
    if kind == "flow_cg":
        n = rng.randint(9, 16)
        return dict(kind="flow_cg", n=n, density=round(0.4 / 2 ** (0.8 * (n - 9)) + 0.002, 4), columns=rng.randint(20, 100))
    if kind == "screen":
        return dict(kind="screen", n=rng.randint(10, 17), density=0.02, respondents=rng.randint(60, 600),
                    draws=int(math.exp(rng.uniform(math.log(100), math.log(4000)))))
    return dict(kind="mlp", width_in=rng.randint(40, 400), hidden=rng.choice([256, 512, 1024]),
                rows=int(math.exp(rng.uniform(math.log(64), math.log(2048)))))


# ------------------------------------------------------------------ inputs, from the seed alone
def _rows(case, seed):
    """Rows of the case's design (which menus are asked belongs to the case) with p_hat of the seed:
    a Dirichlet mixture of random orders, every menu resampled (as mixture_instance makes them)."""
    n = case["n"]
    K, N = (50, 500) if n >= 16 else (20, 200)
    masks = np.arange(1, 1 << n)
    masks = masks[(masks & (masks - 1)) != 0]
    keep = max(2, round(case["density"] * masks.size))
    menus = np.sort(np.random.default_rng(n).choice(masks, size=keep, replace=False)) if keep < masks.size else masks
    rng = np.random.default_rng(seed)
    orders = np.stack([rng.permutation(n) for _ in range(K)])
    weights = rng.dirichlet(np.ones(K))
    p = np.zeros((menus.size, n))
    np.add.at(p, (np.repeat(np.arange(menus.size), K), top_of_orders(n, menus, orders).reshape(-1)), np.tile(weights, menus.size))
    return rows_of(n, menus, rng.multinomial(N, p / p.sum(axis=1, keepdims=True)) / float(N))


def _batch_rows(case, seed):
    menu, alt, p = _rows(case, seed)
    rng = np.random.default_rng([seed, 1])
    return menu, alt, p, np.clip(p[None, :] + rng.normal(0, 0.02, (case["draws"], p.size)), 0.0, 1.0)


def _screen_parts(case, seed):
    panel, (menu, alt, p) = panel_instance(case["n"], case["density"], case["respondents"], 20, 30, seed=seed)
    d = bootstrap.Draws(panel, menu, alt, p, B=case["draws"], weights="multinomial", seed=seed)
    r_n, eps_n, _ = bootstrap.scaling(d.R)
    fit = np.clip(d.p_hat + 0.01 * np.random.default_rng([seed, 2]).standard_normal(d.M), 0.0, 1.0)
    return d, fit, eps_n * r_n


def _price_rows(case, seed):
    """(menus x-major, offsets, float32 residual scores)."""
    n = case["n"]
    if case["menus"] == "pairs":
        i, j = np.triu_indices(n, 1)
        m = (np.int64(1) << i) | (np.int64(1) << j)
        menu, alt = np.repeat(m, 2), np.stack([i, j], 1).reshape(-1)
        p = np.full(menu.size, 0.5)
    else:
        menu, alt, p = _rows(case, seed)
    menus, _, p32, offsets, _ = flow_cg.prepare_choice_data(menu, alt, p, n)
    # the residual of a fitted mixture: mean zero, the size of sampling noise
    return menus, offsets, np.random.default_rng([seed, 3]).normal(0, 0.05, p32.size).astype(np.float32)


def _mlp_parts(case, seed):
    d = [case["width_in"], case["hidden"], case["hidden"], case["hidden"], case["width_in"]]
    g = torch.Generator().manual_seed(seed)
    par = torch.cat([torch.cat([((2 * torch.rand(d[i + 1] * d[i], generator=g) - 1) / math.sqrt(d[i])),
                                0.02 * torch.randn(d[i + 1], generator=g)]) for i in range(len(d) - 1)])
    X = torch.rand(case["rows"], d[0], generator=g)
    return d, par.numpy(), X.numpy(), (X + 0.05 * torch.randn(X.shape, generator=g)).numpy()


def prepare(case, seed):
    kind, n = case["kind"], case.get("n")
    st = dict(case=case)
    if kind in ("solve", "flow_cg"):
        menu, alt, p = _rows(case, seed)
        st.update(rum=RUM(menu, alt, p, num_alternatives=n), p=p)
        if kind == "solve" and not case["tol"]:
            st["session"] = st["rum"].session(method="bm_admm", method_args=dict(dtype=case["dtype"], max_iter=case["iters"]))
    elif kind == "batch":
        menu, alt, p, P = _batch_rows(case, seed)
        ctx = context()
        beta = _beta(p.size)
        prob = ctx.bm_problem(n, menu, alt, p)
        _, _, kept = ctx.bm_solve(prob, ctx.bm_params(beta, max_iter=100, abs_tol=0.0, rel_tol=None, dtype=case["dtype"]),
                                  keep=True)
        par = ctx.bm_params(beta, max_iter=case["iters"], abs_tol=0.0, rel_tol=None, dtype=case["dtype"])
        st.update(ctx=ctx, prob=prob, par=par, P=P, warm=kept)
    elif kind == "price":
        menus, offsets, scores = _price_rows(case, seed)
        st.update(pricer=_lib.Pricer(context(), n, menus, offsets, mode=case["mode"]), scores=scores)
    elif kind == "screen":
        d, fit, scale = _screen_parts(case, seed)
        st.update(rows=_lib.DrawRows(context(), d.W, d.lists, d.p_hat), fit=fit, scale=scale)
    else:
        d, par, X, T = _mlp_parts(case, seed)
        net = _lib.MLP(context(), d)
        net.set_params(par)
        st.update(net=net, X=X, T=T)
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "solve":
        if case["tol"]:
            r = state["rum"].calculate_distance(method="bm_admm", method_args=dict(max_iter=case["iters"]))
        else:
            r = state["session"].solve(state["p"], abs_tol=0.0, rel_tol=0.0)
        # a float32 state's fit is kept as the float32 values it is good for
        f = np.float32 if case["dtype"] == "float32" else np.float64
        return dict(lb=f(r.lb), ub=f(r.ub), p_fit=r.p_fit.astype(f), iterations=r.iterations)
    if kind == "flow_cg":
        r = state["rum"].calculate_distance(method="flow_cg", method_args=dict(max_iters=case["columns"]))
        return dict(lb=r.lb, ub=r.ub, p_fit=r.p_fit, iterations=r.iterations)
    if kind == "batch":
        res, _ = state["ctx"].bm_solve_batch(state["prob"], state["par"], state["P"], warm=state["warm"], want_fit=True)
        return dict(lb=np.array([r["lb"] for r in res]), ub=np.array([r["ub"] for r in res]),
                    p_fit=np.stack([r["p_fit"] for r in res]), iterations=np.array([r["iters"] for r in res]))
    if kind == "price":
        vmax, rank, margin = state["pricer"].price(state["scores"])
        return dict(vmax=vmax, rank=rank, margin=margin)
    if kind == "screen":
        dev, ub = state["rows"].screen(state["fit"], state["scale"])
        return dict(dev=dev, ub=ub)
    loss, grad = state["net"].loss_grad(state["X"], state["T"])
    return dict(loss=loss, grad=grad)


# ------------------------------------------------------------------ work
def _row_count(case):
    return case["density"] * case["n"] * 2 ** (case["n"] - 1) + case["n"]


def work(case):
    """A solve: each iteration reads and writes its two multiplier arrays (one value per
    (alternative, menu) each) once and applies the four butterfly transforms; a pricing sweep: the
    rows' scores and the float32 (or quantized) lattice written once, one addition per qualifying
    (row, subset); a screen: the weights read once, the two norms written."""
    kind, n = case["kind"], case.get("n")
    if kind in ("solve", "batch"):
        S, e = n << (n - 1), 8 if case["dtype"] == "float64" else 4
        it = case["iters"] * case.get("draws", 1)
        return dict(bytes=float(it * 4 * S * e + 24 * _row_count(case)), flops=float(it * S * (n - 1) * 6.5))
    if kind == "price":
        e = {"mask": 5, "f32": 4, "u16": 2, "u24": 3}[case["mode"]]
        if case["menus"] == "pairs":
            mp, adds = n * (n - 1), n * (n - 1) * 2.0 ** (n - 2)
        else:                                  # a menu of k members has k rows, each within 2^(n - k) subsets
            mp = _row_count(case)
            adds = case["density"] * sum(math.comb(n, k) * k * 2.0 ** (n - k) for k in range(2, n + 1))
        return dict(bytes=4.0 * mp + e * 2.0 ** n, flops=adds + n * 2.0 ** (n - 1))
    if kind == "flow_cg":
        mp = _row_count(case)
        adds = case["density"] * sum(math.comb(n, k) * k * 2.0 ** (n - k) for k in range(2, n + 1))
        return dict(bytes=case["columns"] * (20 * mp + 5 * 2.0 ** n), flops=case["columns"] * (adds + n * 2.0 ** (n - 1)))
    if kind == "screen":
        B, R = case["draws"], case["respondents"]
        M = min(R * 20.0 * case["n"] / 2, _row_count(case))
        return dict(bytes=8.0 * B * R + 16.0 * B + 24.0 * M, flops=B * (4.0 * R * 20 + 6.0 * M))
    d = [case["width_in"], case["hidden"], case["hidden"], case["hidden"], case["width_in"]]
    mults = sum(d[i] * d[i + 1] for i in range(4))
    return dict(bytes=8.0 * case["rows"] * d[0] + 8.0 * mults, flops=6.0 * case["rows"] * mults)


# ------------------------------------------------------------------ the same in 64 bits
def _beta(mp):
    return min(100.0, max(0.3, 10 ** -1.48 * float(mp) ** 0.508))


def _fly(v, n, a, b, c, d):
    """The 2x2 butterfly (a, b; c, d) over the n - 1 rest bits of every alternative's block."""
    shape = v.shape
    for j in range(n - 1):
        w = v.reshape(-1, 2, 1 << j)
        lo, hi = w[:, 0], w[:, 1]
        v = torch.stack((a * lo + b * hi, c * lo + d * hi), 1)
    return v.reshape(shape)


class _Admm:
    """The BM-ADMM iteration and its certificate on dense float64 tensors (draws x slab)."""

    def __init__(self, n, menu, alt, P, beta):
        dev = "cuda"
        self.n, self.N, self.Nl, self.b = n, 1 << n, 1 << (n - 1), beta
        self.P = torch.as_tensor(np.atleast_2d(P), dtype=torch.float64, device=dev)
        menu, alt = torch.as_tensor(menu, device=dev).long(), torch.as_tensor(alt, device=dev).long()
        rest = menu & ~(torch.ones_like(menu) << alt)
        self.obs = alt * self.Nl + self._compress(rest, alt)
        xh = torch.zeros(self.P.shape[0], n * self.Nl, dtype=torch.float64, device=dev)
        xh[:, self.obs] = self.P
        self.w = torch.zeros(n * self.Nl, dtype=torch.bool, device=dev)
        self.w[self.obs] = True
        self.xh = xh
        G = np.array([[1.0, -1.0], [-1.0, 1.0 + P_COND ** 2]])
        self.ev, self.Q = np.linalg.eigh(G)
        pc = sum((torch.arange(self.Nl, device=dev) >> j) & 1 for j in range(n - 1))
        self.diag = (1.0 / (1.0 + self.ev[1] ** pc.double() * self.ev[0] ** (n - 1 - pc).double())).repeat(n)
        S = torch.arange(self.N, device=dev)
        self.size = sum((S >> i) & 1 for i in range(n))
        self.mw = torch.zeros(self.N, dtype=torch.int32, device=dev)           # observed members of each menu
        for i in range(n):
            m = ((S >> i) & 1).bool()
            self.mw[m] += self.w[i * self.Nl:(i + 1) * self.Nl].int()
        self.x2 = self._prox(xh)
        self.s = torch.zeros_like(xh)
        self.y = torch.zeros_like(xh)
        self.z = torch.zeros_like(xh)

    @staticmethod
    def _compress(rest, x):
        low = (torch.ones_like(rest) << x) - 1
        return (rest & low) | ((rest >> (x + 1)) << x)

    def _blocks(self, v, i):
        """Alternative i's block spread over the menus with i (2^i-strided pairs): a view of v."""
        return v[:, i * self.Nl:(i + 1) * self.Nl].reshape(v.shape[0], -1, 1 << i)

    def _over(self, arr, i):
        """The entries of a per-menu array at the menus containing i, in the block's order."""
        return arr.reshape(arr.shape[0], -1, 2, 1 << i)[:, :, 1]

    def _prox(self, v):
        B, b = v.shape[0], self.b
        c = b + 2.0 * self.w.double()
        t = b * v + 2.0 * self.w * self.xh
        tau = torch.full((B, self.N), -1e300, dtype=torch.float64, device=v.device)
        last = None
        for _ in range(self.n + 2):                # the active set only shrinks
            num = torch.full((B, self.N), -1.0, dtype=torch.float64, device=v.device)
            den = torch.zeros_like(num)
            for i in range(self.n):
                ti, ci = self._blocks(t, i), self._blocks(c[None], i)
                on = ti > self._over(tau, i)
                self._over(num, i).add_(torch.where(on, ti / ci, 0.0))
                self._over(den, i).add_(torch.where(on, 1.0 / ci, 0.0))
            new = torch.where(den > 0, num / den, tau)
            if last is not None and torch.equal(new, last):
                break
            last = tau = new
        u = torch.empty_like(v)
        for i in range(self.n):
            self._blocks(u, i).copy_(torch.clamp((self._blocks(t, i) - self._over(tau, i)) / self._blocks(c[None], i), min=0))
        return u

    def iterate(self):
        n, b, Q, p = self.n, self.b, self.Q, P_COND
        v = _fly(self.y - b * self.s, n, 1.0, 0.0, -1.0, p)
        v = _fly((self.z + b * self.x2 - v) / b, n, Q[0, 0], Q[1, 0], Q[0, 1], Q[1, 1]) * self.diag
        x = _fly(v, n, Q[0, 0], Q[0, 1], Q[1, 0], Q[1, 1])
        ax = _fly(x, n, 1.0, -1.0, 0.0, p)
        a = -ALPHA * ax - (1 - ALPHA) * self.s
        self.s = torch.clamp(self.y / b - a, min=0)
        self.y = self.y - b * (a + self.s)
        xo = ALPHA * x + (1 - ALPHA) * self.x2
        self.x2 = self._prox(xo - self.z / b)
        self.z = self.z - b * (xo - self.x2)

    def check(self):
        """(ub, lb, the pushed point on the rows) of every draw."""
        n, B, eps = self.n, self.P.shape[0], 1e-12
        w = torch.clamp(_fly(self.x2, n, 1.0, -1.0, 0.0, 1.0), min=0) + eps
        out = torch.zeros(B, self.N, dtype=torch.float64, device=w.device)
        for i in range(n):                         # outflow of D: over the x not in D, entry (x, D)
            out.reshape(B, -1, 2, 1 << i)[:, :, 0].add_(self._blocks(w, i))
        mass = torch.zeros_like(out)
        mass[:, 0] = 1.0
        for k in range(n):                         # layer k's masses go out to layer k + 1
            src = torch.where((self.size == k) & (out > 0), mass / torch.where(out > 0, out, 1.0), 0.0)
            for i in range(n):
                self._over(mass, i).add_(src.reshape(B, -1, 2, 1 << i)[:, :, 0] * self._blocks(w, i))
        ratio = torch.where(out > 0, mass / torch.where(out > 0, out, 1.0), 0.0)
        for i in range(n):
            self._blocks(w, i).mul_(ratio.reshape(B, -1, 2, 1 << i)[:, :, 0])
        fit = _fly(w, n, 1.0, 1.0, 0.0, 1.0)[:, self.obs]
        ub = (fit - self.P).square().sum(1).sqrt()
        y = self.x2[:, self.obs]
        r = self.P - y
        g = torch.zeros_like(self.x2)
        g[:, self.obs] = r
        g = _fly(g, n, 1.0, 0.0, 1.0, 1.0)
        dp = torch.full((B, self.N), -1e300, dtype=torch.float64, device=w.device)
        dp[:, 0] = 0.0
        for k in range(1, n + 1):
            src = torch.where(self.size == k - 1, dp, -1e300)
            for i in range(n):
                tgt = self._over(dp, i)
                torch.maximum(tgt, src.reshape(B, -1, 2, 1 << i)[:, :, 0] + self._blocks(g, i), out=tgt)
        lb2 = r.square().sum(1) - 2.0 * (dp[:, -1] - (r * y).sum(1))
        return ub, torch.clamp(lb2, min=0).sqrt(), fit

    def solve(self, iters, abs_tol=0.0, rel_tol=0.0, check=50):
        ub = torch.full((self.P.shape[0],), math.inf, dtype=torch.float64, device=self.P.device)
        lb, fit, it = torch.zeros_like(ub), torch.zeros_like(self.P), 0
        while it < iters:
            for _ in range(check):
                self.iterate()
            it += check
            u, low, f = self.check()
            fit = torch.where((u < ub)[:, None], f, fit)
            ub, lb = torch.minimum(ub, u), torch.maximum(lb, low)
            if bool(((ub - lb <= abs_tol) | (ub - lb <= rel_tol * lb)).all()):
                break
        return ub.cpu().numpy(), lb.cpu().numpy(), fit.cpu().numpy(), it


def _exact_price(case, seed):
    n = case["n"]
    if n > 24:
        return None                                # the float64 sums of every (x, subset) pass 10 GB
    menus, offsets, scores = _price_rows(case, seed)
    Nl, N = 1 << (n - 1), 1 << n
    x = np.repeat(np.arange(n), np.diff(offsets))
    rest = menus.astype(np.int64) & ~(np.int64(1) << x)
    pos = x * Nl + ((rest & ((np.int64(1) << x) - 1)) | ((rest >> (x + 1)) << x))
    w = torch.zeros(n * Nl, dtype=torch.float64, device="cuda")
    w.index_add_(0, torch.as_tensor(pos, device="cuda"), torch.as_tensor(scores, device="cuda").double())
    w = _fly(w[None], n, 1.0, 0.0, 1.0, 1.0)[0]
    S = torch.arange(N, device="cuda")
    size = sum((S >> i) & 1 for i in range(n))
    dp = torch.full((N,), -1e300, dtype=torch.float64, device="cuda")
    dp[0] = 0.0
    for k in range(1, n + 1):
        src = torch.where(size == k - 1, dp, -1e300)
        for i in range(n):
            tgt = dp.reshape(-1, 2, 1 << i)[:, 1]
            torch.maximum(tgt, src.reshape(-1, 2, 1 << i)[:, 0] + w[i * Nl:(i + 1) * Nl].reshape(-1, 1 << i), out=tgt)
    return dict(vmax=float(dp[-1]), rank=None, margin=None)


def _exact_screen(case, seed):
    d, fit, scale = _screen_parts(case, seed)
    L, R = d.lists, d.R
    dev = "cuda"
    W = torch.as_tensor(d.W, dtype=torch.float64, device=dev)

    def dense(ptr, resp, cnt):
        m = torch.zeros(len(ptr) - 1, R, dtype=torch.float64, device=dev)
        at = torch.as_tensor(np.repeat(np.arange(len(ptr) - 1), np.diff(ptr)), device=dev)
        m.index_put_((at, torch.as_tensor(np.asarray(resp), device=dev).long()),
                     torch.as_tensor(np.asarray(cnt), dtype=torch.float64, device=dev), accumulate=True)
        return m

    offered = dense(np.asarray(L.menu_ptr), L.menu_resp, L.menu_cnt)
    chose = dense(np.asarray(L.row_ptr), L.row_resp, L.row_cnt)
    at = torch.as_tensor(np.asarray(L.row_menu), device=dev).long()
    p, f = torch.as_tensor(d.p_hat, device=dev), torch.as_tensor(fit, device=dev)
    out = [[], []]
    for b in range(0, W.shape[0], 256):
        seen, got = (W[b:b + 256] @ offered.T)[:, at], W[b:b + 256] @ chose.T
        q = torch.where(seen > 0, got / torch.where(seen > 0, seen, 1.0), p) - p
        out[0].append(q.square().sum(1).sqrt())
        out[1].append((p + scale * q - f).square().sum(1).sqrt())
    return dict(dev=torch.cat(out[0]).cpu().numpy(), ub=torch.cat(out[1]).cpu().numpy())


def _exact_mlp(case, seed):
    d, par, X, T = _mlp_parts(case, seed)
    par = torch.as_tensor(par, device="cuda").double().requires_grad_()
    h, at = torch.as_tensor(X, device="cuda").double(), 0
    for i in range(len(d) - 1):
        W = par[at:at + d[i] * d[i + 1]].reshape(d[i + 1], d[i])
        at += d[i] * d[i + 1]
        h = h @ W.T + par[at:at + d[i + 1]]
        at += d[i + 1]
        if i + 2 < len(d):
            h = torch.nn.functional.gelu(h)
    loss = (h - torch.as_tensor(T, device="cuda").double()).square().mean()
    loss.backward()
    return dict(loss=float(loss.detach()), grad=par.grad.cpu().numpy())


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        menu, alt, p = _rows(case, seed)
        a = _Admm(case["n"], menu, alt, p, _beta(p.size))
        ub, lb, fit, it = a.solve(case["iters"], *((1e-5, 1e-4) if case["tol"] else (0.0, 0.0)))
        if case["dtype"] == "float32":             # the bounds certify the float32 iterate itself: no value of their own
            return dict(lb=None, ub=None, p_fit=fit[0], iterations=None)
        return dict(lb=float(lb[0]), ub=float(ub[0]), p_fit=fit[0], iterations=None)
    if kind == "batch":
        menu, alt, p, P = _batch_rows(case, seed)
        a = _Admm(case["n"], menu, alt, p, _beta(p.size))
        for _ in range(100):
            a.iterate()
        b = _Admm(case["n"], menu, alt, P, _beta(p.size))
        b.x2, b.s, b.y, b.z = (t.expand(P.shape[0], -1).clone() for t in (a.x2, a.s, a.y, a.z))
        ub, lb, fit, _ = b.solve(case["iters"])
        return dict(lb=lb, ub=ub, p_fit=fit, iterations=None)
    if kind == "price":
        return _exact_price(case, seed)
    if kind == "screen":
        return _exact_screen(case, seed)
    if kind == "mlp":
        return _exact_mlp(case, seed)
    return None                                    # flow_cg: its columns follow float32 pricing values
