"""The workloads the engine's speed is judged by: what a program that uses this
framework has it do, through its public entry points.

Three kinds of case:

  solve    one LP through ``Engine.solve`` (with ``fresh``, ``Engine.load`` first:
           a new LP on an engine the program keeps);
  batch    many LPs through ``Engine.solve_batch`` (with ``fresh``,
           ``Engine.load_batch`` first);
  network  one training batch of the warm start's network: ``Mlp.forward`` and
           ``Mlp.gradients``.

The LPs are the seeded families of ``lpgen`` (the repository's benchmark and
tests run on them). ``form`` says which iteration a program asks for:

  reference  the defaults (the reference's own rules, precision fp64_exact);
  averaged   restarted averaged PDHG: relative_kkt_l2, adaptive_l2 restarts;
  halpern    the reflected Halpern iteration on the same rules.

Every solve runs a fixed budget of iterations (the tolerance of the last two
forms is out of reach), so that a pass is the same work whatever the rounding.
"""
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("sovereign-solver_b200")

PERIOD = 40          # PdhgOptions.restart_check_period
ON_CHIP = 126e6      # bytes of L2: a matrix that fits is read from HBM once


def listed():
    return [
        # the smallest drop-in call: Pdhg.solve on a toy LP, the reference's
        # defaults (setup and launches count as much as iterations)
        dict(name="exact_toy_60x150_fresh", kind="solve", family="equality", m=60, n=150, k=4,
             precision="fp64_exact", form="reference", weight=False, iters=400, fresh=True),
        # an ordinary drop-in call: the repository's 2,000 x 5,000 LP
        dict(name="exact_2000x5000_fresh", kind="solve", family="equality", m=2000, n=5000, k=5,
             precision="fp64_exact", form="reference", weight=False, iters=1000, fresh=True),
        # the drop-in on a network LP with long rows, solved again from residence
        dict(name="exact_transport_200x501", kind="solve", family="transportation", m=200, n=501,
             k=2, precision="fp64_exact", form="reference", weight=False, iters=300, fresh=False),
        # a small LP at the warm-start family's base size: many are solved in turn
        dict(name="mixed_equality_500x1200", kind="solve", family="equality", m=500, n=1200, k=5,
             precision="mixed", form="halpern", weight=True, iters=800, fresh=False),
        # a mid-size LP in full precision, odd sizes, averaged form
        dict(name="fp64_equality_20011x50021", kind="solve", family="equality", m=20011, n=50021,
             k=5, precision="fp64", form="averaged", weight=True, iters=400, fresh=False),
        # a mid-size network LP, odd sizes, budget not a multiple of the period
        dict(name="fp64_transport_701x1499", kind="solve", family="transportation", m=701, n=1499,
             k=2, precision="fp64", form="averaged", weight=False, iters=210, fresh=False),
        # a new LP end to end: load, scale, solve (the large warm-start base's size)
        dict(name="mixed_equality_50000x120000_fresh", kind="solve", family="equality", m=50000,
             n=120000, k=5, precision="mixed", form="halpern", weight=True, iters=200, fresh=True),
        # the badly scaled LP of the precision study, its FP64 arm
        dict(name="fp64_badly_200000x500000", kind="solve", family="badly_scaled", m=200000,
             n=500000, k=8, precision="fp64", form="halpern", weight=True, iters=400,
             fresh=False),
        # the headline: ten million columns, twenty million nonzeros
        dict(name="mixed_transport_2000x5000", kind="solve", family="transportation", m=2000,
             n=5000, k=2, precision="mixed", form="halpern", weight=False, iters=600,
             fresh=False),
        # a batch of uneven LPs, resident
        dict(name="batch_mixed_256_uneven", kind="batch", count=256, m_lo=50, m_hi=5000, k=0,
             precision="mixed", form="halpern", weight=True, iters=200, fresh=False),
        # a small batch of equal LPs, loaded and solved
        dict(name="batch_fp64_67_even_fresh", kind="batch", count=67, m_lo=500, m_hi=500, k=5,
             precision="fp64", form="averaged", weight=True, iters=200, fresh=True),
        # one training batch of the warm-start network
        dict(name="network_256", kind="network", rows=256, n_in=64, hidden=512, n_out=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


MOST_WORK = 20e6 * 600  # nonzeros x iterations of the largest listed case


def draw(rng):
    pick = rng.random()
    if pick < 0.06:
        return dict(kind="network", rows=8 * rng.randint(1, 64), n_in=64, hidden=512, n_out=512)
    precision = rng.choice(["fp64_exact", "mixed", "fp64", "mixed", "fp64"])
    if pick < 0.30:
        if precision == "fp64_exact":
            precision = "fp64"
        m_lo = _log_int(rng, 50, 500)
        return dict(kind="batch", count=_log_int(rng, 8, 300), m_lo=m_lo,
                    m_hi=_log_int(rng, m_lo, 5000), k=rng.choice([0, 4, 5, 7]),
                    precision=precision, form=rng.choice(["averaged", "halpern"]), weight=True,
                    iters=_log_int(rng, 80, 320), fresh=rng.random() < 0.4)
    form = "reference" if precision == "fp64_exact" else rng.choice(["averaged", "halpern"])
    family = rng.choice(["equality", "transportation", "badly_scaled"])
    if family == "transportation":
        m = _log_int(rng, 10, 2000)
        n = int(m * rng.uniform(1.5, 2.5)) + 1
        k, nnz, weight = 2, 2 * m * n, False
    else:
        m = _log_int(rng, 50, 200000)
        n = int(m * rng.uniform(2.0, 3.0)) + 1
        k = rng.randint(4, 8)
        nnz, weight = n * k, True
    if precision == "fp64_exact":
        weight = False
    iters = _log_int(rng, 120, 900)
    iters = max(41, min(iters, int(MOST_WORK / nnz)))
    if nnz > 200000:  # large LPs: fewer iterations, as the listed ones
        iters = min(iters, 600 if family == "transportation" else 400)
    if precision == "mixed" and family == "badly_scaled":
        # FP32 iterates of this family part from the 64-bit ones within a few
        # hundred iterations on small LPs: large ones and a short budget
        if m < 20000:
            family = "equality"
        else:
            iters = min(iters, 80)
    return dict(kind="solve", family=family, m=m, n=n, k=k, precision=precision, form=form,
                weight=weight, iters=iters, fresh=rng.random() < 0.4)


# ---- inputs --------------------------------------------------------------------


def _problem(case, seed):
    L = pkg.lpgen
    if case["family"] == "equality":
        return L.random_equality_lp(case["m"], case["n"], case["k"], seed=seed)
    if case["family"] == "transportation":
        return L.transportation_lp(case["m"], case["n"], seed=seed)
    return L.badly_scaled_lp(case["m"], case["n"], case["k"], seed=seed)


def _batch_shapes(case):
    """(rows, columns, entries per column) of each instance: rows spread
    evenly over the logarithm, columns 2 or 3 times as many."""
    lo, hi, count = math.log(case["m_lo"]), math.log(case["m_hi"]), case["count"]
    out = []
    for i in range(count):
        m = int(math.exp(lo + (hi - lo) * i / max(1, count - 1)) + 1e-9)
        out.append((m, m * (2 + i % 2), case["k"] or 4 + i % 7))
    return out


def _problems(case, seed):
    shapes = _batch_shapes(case)
    order = np.random.default_rng(seed).permutation(len(shapes))
    return [pkg.lpgen.random_equality_lp(*shapes[i], seed=1000 * seed + int(i)) for i in order]


def _options(case):
    o = dict(precision=case["precision"], max_iterations=case["iters"])
    if case["form"] != "reference":
        o.update(tolerance=1e-11, termination_rule="relative_kkt_l2", restart_rule="adaptive_l2",
                 primal_weight_update=case["weight"], halpern=case["form"] == "halpern")
    return pkg.PdhgOptions(**o)


def _network_inputs(case, seed):
    rng = np.random.default_rng(seed)
    d = (case["n_in"], case["hidden"], case["hidden"], case["n_out"])
    parts = []
    for a, b in zip(d[:-1], d[1:]):
        parts.append((rng.standard_normal((b, a)) * math.sqrt(2.0 / a)).astype(np.float32))
        parts.append((rng.standard_normal(b) * 0.1).astype(np.float32))
    x = (rng.standard_normal((case["rows"], case["n_in"])) * 0.1).astype(np.float32)
    t = rng.standard_normal((case["rows"], case["n_out"])).astype(np.float32)
    return parts, x, t


def prepare(case, seed):
    if case["kind"] == "network":
        parts, x, t = _network_inputs(case, seed)
        net = pkg.mlp.Mlp(case["n_in"], case["hidden"], case["n_out"])
        net.set_params(np.concatenate([p.ravel() for p in parts]))
        return dict(case=case, net=net, x=x, t=t)
    engine = pkg.Engine(0)
    if case["kind"] == "batch":
        problems = _problems(case, seed)
        if not case["fresh"]:
            engine.load_batch(problems)
    else:
        problems = _problem(case, seed)
        if not case["fresh"]:
            engine.load(problems)
    return dict(case=case, engine=engine, problems=problems, options=_options(case))


# ---- one pass ------------------------------------------------------------------


def _point(case, v):
    """A point as the program goes on with it: a mixed solve's carries FP32
    precision (the network trains on it in FP32)."""
    t = torch.from_numpy(v)
    return t.float() if case["precision"] == "mixed" else t


def run(state):
    case = state["case"]
    if case["kind"] == "network":
        y = state["net"].forward(state["x"])
        g, loss = state["net"].gradients(state["x"], state["t"])
        return dict(y=y, gradients=g, loss=loss)
    engine, opt = state["engine"], state["options"]
    if case["kind"] == "solve":
        if case["fresh"]:
            engine.load(state["problems"])
        r = engine.solve(opt)
        out = dict(primal=_point(case, r.primal), dual=_point(case, r.dual),
                   reduced_costs=_point(case, r.reduced_costs), objective=r.objective,
                   iterations=r.iterations, restarts=r.restarts)
        if case["precision"] != "mixed":  # an FP32 point's residual is its rounding
            out["relative_kkt"] = r.relative_kkt
        return out
    if case["fresh"]:
        engine.load_batch(state["problems"])
    rs = engine.solve_batch(opt)
    return dict(primal=_point(case, np.concatenate([r.primal for r in rs])),
                dual=_point(case, np.concatenate([r.dual for r in rs])),
                reduced_costs=_point(case, np.concatenate([r.reduced_costs for r in rs])),
                objective=np.array([r.objective for r in rs]).astype(
                    np.float32 if case["precision"] == "mixed" else np.float64),
                iterations=np.array([r.iterations for r in rs]),
                restarts=np.array([r.restarts for r in rs]))


# ---- what a pass cannot do without ----------------------------------------------


def work(case):
    if case["kind"] == "network":
        w = case["n_in"] * case["hidden"] + case["hidden"] ** 2 + case["hidden"] * case["n_out"]
        # forward twice (once on its own), backward two products per layer but the first's input
        f = 2.0 * case["rows"] * (4 * w - case["n_in"] * case["hidden"])
        b = 4.0 * (2 * w + case["rows"] * (2 * case["n_in"] + 2 * case["n_out"]))
        return dict(bytes=b, flops=f)
    if case["kind"] == "batch":
        shapes = _batch_shapes(case)
        m, n = sum(s[0] for s in shapes), sum(s[1] for s in shapes)
        nnz = sum(s[1] * s[2] for s in shapes)
    elif case["family"] == "transportation":
        m, n = case["m"] + case["n"], case["m"] * case["n"]
        nnz = 2 * n
    else:
        m, n, nnz = case["m"], case["n"], case["n"] * case["k"]
    vb = 4.0 if case["precision"] == "mixed" else 8.0
    matrix = (vb + 4.0) * nnz
    # the LP read once and the point written once; a matrix beyond the L2 again
    # by both products of every iteration
    once = matrix + 8.0 * (3 * n + 2 * m) + 8.0 * (2 * n + m)
    again = 2.0 * vb * nnz * case["iters"] if matrix > ON_CHIP else 0.0
    return dict(bytes=once + again, flops=4.0 * nnz * case["iters"])


# ---- the same in plain 64-bit tensors ---------------------------------------------


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Lps:
    """LPs stacked block-diagonally as FP64 tensors; ri / ci: each row's and
    column's LP."""

    def __init__(self, problems):
        d = _dev()
        cat = lambda f: torch.from_numpy(np.concatenate([f(p) for p in problems])).to(d)  # noqa: E731
        self.count = len(problems)
        ms, ns = [p.m for p in problems], [p.n for p in problems]
        r0, c0 = np.cumsum([0] + ms), np.cumsum([0] + ns)
        self.m, self.n = int(r0[-1]), int(c0[-1])
        lengths = np.concatenate([np.diff(p.row_ptr) for p in problems]).astype(np.int64)
        self.rp = torch.from_numpy(np.concatenate([[0], np.cumsum(lengths)])).to(d)
        self.col = torch.from_numpy(np.concatenate(
            [p.col_idx.astype(np.int64) + o for p, o in zip(problems, c0)])).to(d)
        self.row = torch.repeat_interleave(torch.arange(self.m, device=d),
                                           torch.from_numpy(lengths).to(d))
        self.val = cat(lambda p: p.val)
        self.c, self.lo, self.hi = cat(lambda p: p.c), cat(lambda p: p.col_lo), cat(lambda p: p.col_hi)
        self.rlo, self.rhi = cat(lambda p: p.row_lo), cat(lambda p: p.row_hi)
        self.ri = torch.repeat_interleave(torch.arange(self.count, device=d), torch.tensor(ms, device=d))
        self.ci = torch.repeat_interleave(torch.arange(self.count, device=d), torch.tensor(ns, device=d))
        order = torch.sort(self.col, stable=True)[1]
        self.t_col, self.t_order = self.row[order], order
        counts = torch.bincount(self.col, minlength=self.n)
        self.t_rp = torch.cat([torch.zeros(1, dtype=torch.int64, device=d), counts.cumsum(0)])

    def products(self, val):
        """x -> A x and y -> A^T y with the values `val`."""
        if self.row.is_cuda:
            a = torch.sparse_csr_tensor(self.rp, self.col, val, (self.m, self.n))
            t = torch.sparse_csr_tensor(self.t_rp, self.t_col, val[self.t_order], (self.n, self.m))
            return (lambda x: torch.mv(a, x)), (lambda y: torch.mv(t, y))
        zero = lambda k: torch.zeros(k, dtype=torch.float64)  # noqa: E731
        return (lambda x: zero(self.m).index_add_(0, self.row, val * x[self.col]),
                lambda y: zero(self.n).index_add_(0, self.col, val * y[self.row]))

    def total(self, by, v):
        return torch.zeros(self.count, dtype=torch.float64, device=v.device).index_add_(0, by, v)

    def top(self, by, v, size=None):
        z = torch.zeros(size or self.count, dtype=torch.float64, device=v.device)
        return z.scatter_reduce_(0, by, v, "amax", include_self=True)


def _clamp(v, lo, hi):
    return torch.minimum(torch.maximum(v, lo), hi)


def _sign_violation(v, lo, hi):
    """The part of a multiplier outside the sign that its bounds allow."""
    fl, fh = torch.isfinite(lo), torch.isfinite(hi)
    one = torch.where(fl, torch.clamp(-v, min=0), torch.clamp(v, min=0))
    return torch.where(fl & fh, torch.zeros_like(v), torch.where(fl | fh, one, v.abs()))


def _beyond(act, lo, hi):
    return torch.clamp(torch.maximum(lo - act, act - hi), min=0)


def _active_term(v, act, lo, hi, tol):
    """A multiplier's contribution under the reference's activity test."""
    at_lo, at_hi = (act - lo).abs() < tol, (act - hi).abs() < tol
    r = torch.where(at_lo & ~at_hi, torch.clamp(-v, min=0), torch.clamp(v, min=0))
    return torch.where(at_lo & at_hi, torch.zeros_like(v), torch.where(at_lo | at_hi, r, v.abs()))


def _finite_product(v, lo, hi):
    t = torch.where(v > 0, lo, hi)
    return torch.where(torch.isfinite(t), v * torch.where(torch.isfinite(t), t, torch.zeros_like(t)),
                       torch.zeros_like(v))


def _pdhg(S, case):
    """The documented algorithm on every LP of S: Ruiz and Pock-Chambolle
    scaling, the power iteration's step, the iteration, restarts."""
    f64 = dict(dtype=torch.float64, device=S.val.device)
    ri, ci = S.ri, S.ci
    rs, cs = torch.ones(S.m, **f64), torch.ones(S.n, **f64)
    a = S.val.abs()
    open_ = torch.ones(S.count, dtype=torch.bool, device=S.val.device)
    for _ in range(8):
        v = a * rs[S.row] * cs[S.col]
        rm, cm = S.top(S.row, v, S.m), S.top(S.col, v, S.n)
        rs = torch.where((rm > 0) & open_[ri], rs / torch.where(rm > 0, rm, 1.0).sqrt(), rs)
        cs = torch.where((cm > 0) & open_[ci], cs / torch.where(cm > 0, cm, 1.0).sqrt(), cs)
        worst = torch.maximum(S.top(ri, torch.where(rm > 0, (rm - 1).abs(), 0.0)),
                              S.top(ci, torch.where(cm > 0, (cm - 1).abs(), 0.0)))
        open_ = open_ & ~(worst < 1e-2)
    v = a * rs[S.row] * cs[S.col]
    rsum = torch.zeros(S.m, **f64).index_add_(0, S.row, v)
    csum = torch.zeros(S.n, **f64).index_add_(0, S.col, v)
    rs = torch.where(rsum > 0, rs / torch.where(rsum > 0, rsum, 1.0).sqrt(), rs)
    cs = torch.where(csum > 0, cs / torch.where(csum > 0, csum, 1.0).sqrt(), cs)
    mul, mul_t = S.products(S.val * rs[S.row] * cs[S.col])
    c, lo, hi = S.c * cs, S.lo / cs, S.hi / cs
    rlo, rhi = S.rlo * rs, S.rhi * rs

    u, q = torch.ones(S.n, **f64), torch.ones(S.m, **f64)
    for _ in range(30):
        w = q - mul(u)
        w = w / S.total(ri, w * w).sqrt()[ri]
        u = -mul_t(w)
        est = (S.total(ci, u * u) + S.total(ri, w * w)).sqrt()
        u, q = u / est[ci], w / est[ri]
    eta = 0.9 / est

    def larger(l, h):  # noqa: E741
        z = torch.zeros_like(l)
        return torch.maximum(torch.where(torch.isfinite(l), l.abs(), z),
                             torch.where(torch.isfinite(h), h.abs(), z))

    halpern, rule2 = case["form"] == "halpern", case["form"] != "reference"
    omega = torch.ones(S.count, **f64)
    if case["weight"]:
        omega = S.total(ci, c * c).sqrt() / S.total(ri, larger(rlo, rhi) ** 2).sqrt()
    bnorm = S.total(ri, larger(S.rlo, S.rhi) ** 2).sqrt()
    cnorm = S.total(ci, S.c ** 2).sqrt()
    x, y = _clamp(torch.zeros(S.n, **f64), lo, hi), torch.zeros(S.m, **f64)
    s = _clamp(torch.zeros(S.m, **f64), rlo, rhi)
    xs, ys = torch.zeros_like(x), torch.zeros_like(y)  # sums, or T(z)
    xa, sa, ya = x, s, y
    xl, yl = x, y
    inf = torch.full((S.count,), math.inf, **f64)
    last, prev = inf.clone(), inf.clone()
    since = torch.zeros(S.count, **f64)
    restarts = torch.zeros(S.count, dtype=torch.int64, device=S.val.device)
    rel = torch.zeros(S.count, **f64)

    def measure(px, py):
        """(restart measure, relative KKT) of a scaled point."""
        act, aty = mul(px), mul_t(py)
        if not rule2:  # the reference's: scaled max-norm terms
            tol = 1e-4
            return torch.maximum(
                S.top(ri, torch.maximum(_beyond(act, rlo, rhi), _active_term(py, act, rlo, rhi, tol))),
                S.top(ci, _active_term(c - aty, px, lo, hi, tol))), torch.zeros(S.count, **f64)
        ao, yo, ro, xo = act / rs, py * rs, (c - aty) / cs, px * cs
        p = S.total(ri, _beyond(ao, S.rlo, S.rhi) ** 2).sqrt() / (1 + bnorm)
        d = (S.total(ri, _sign_violation(yo, S.rlo, S.rhi) ** 2)
             + S.total(ci, _sign_violation(ro, S.lo, S.hi) ** 2)).sqrt() / (1 + cnorm)
        po = S.total(ci, S.c * xo)
        do = S.total(ri, _finite_product(yo, S.rlo, S.rhi)) + S.total(ci, _finite_product(ro, S.lo, S.hi))
        g = (po - do).abs() / (1 + po.abs() + do.abs())
        return (p * p + d * d + g * g).sqrt(), torch.maximum(torch.maximum(p, d), g)

    fresh = True
    for it in range(case["iters"]):
        tau_c, tau_r, sig = (eta / omega)[ci], (eta / omega)[ri], (eta * omega)[ri]
        xn = _clamp(x - tau_c * (c - mul_t(y)), lo, hi)
        xb = 2 * xn - x
        sn = _clamp(s - tau_r * y, rlo, rhi)
        sb = 2 * sn - s
        yn = y + sig * (sb - mul(xb))
        if halpern:
            k = since + it % PERIOD
            w = (k + 1) / (k + 2)
            wc, wr = w[ci], w[ri]
            xs, ys = xn, yn
            y = wr * (2 * yn - y) + (1 - wr) * ya
            x, s = wc * xb + (1 - wc) * xa, wr * sb + (1 - wr) * sa
        else:
            x, s, y = xn, sn, yn
            xs, ys = (xn, yn) if fresh else (xs + xn, ys + yn)
        fresh = False
        if (it + 1) % PERIOD:
            continue
        span = since + PERIOD
        if halpern:
            px, py = xs, ys
            cur, rel = measure(px, py)
            cand, to_avg = cur, torch.ones(S.count, dtype=torch.bool, device=x.device)
        else:
            px, py = xs / span[ci], ys / span[ri]
            (cur, rc), (avg, ra) = measure(x, y), measure(px, py)
            to_avg = avg <= cur
            cand, rel = torch.where(to_avg, avg, cur), torch.where(to_avg, ra, rc)
        last = torch.where(torch.isfinite(last), last, cur)
        if rule2:
            go = (cand <= 0.2 * last) | ((cand <= 0.8 * last) & (cand > prev)) | (span >= 0.36 * (it + 1))
            prev, last = cand, torch.where(go, cand, last)
        else:
            to_avg = torch.ones_like(to_avg)
            go = avg <= 0.5 * last
            last = torch.where(go, avg, last)
        restarts += go
        since = torch.where(go, torch.zeros_like(span), span)
        gc, gr = go[ci], go[ri]
        mc, mr = gc & to_avg[ci], gr & to_avg[ri]
        x = torch.where(mc, _clamp(px, lo, hi), x)
        y = torch.where(mr, py, y)
        s = torch.where(mr, _clamp(mul(px), rlo, rhi), s)
        if halpern:
            xa, ya, sa = torch.where(gc, x, xa), torch.where(gr, y, ya), torch.where(gr, s, sa)
        else:
            xs, ys = torch.where(gc, 0.0, xs), torch.where(gr, 0.0, ys)
        if case["weight"]:
            dx, dy = S.total(ci, (x - xl) ** 2).sqrt(), S.total(ri, (y - yl) ** 2).sqrt()
            ok = go & (dx > 1e-10) & (dy > 1e-10)
            omega = torch.where(ok, (omega * dy / torch.where(ok, dx, 1.0)).sqrt(), omega)
            xl, yl = torch.where(gc, x, xl), torch.where(gr, y, yl)
    if halpern:
        x, y = xs, ys
    x, y = x * cs, y * rs
    _, orig_t = S.products(S.val)
    return x, y, S.c - orig_t(y), S.total(ci, S.c * x), rel, restarts


def exact(case, seed):
    if case["kind"] == "network":
        parts, x, t = _network_inputs(case, seed)
        p = [torch.from_numpy(v).double().requires_grad_() for v in parts]
        h = torch.from_numpy(x).double()
        for i in range(3):
            h = h @ p[2 * i].T + p[2 * i + 1]
            h = torch.relu(h) if i < 2 else h
        loss = (h - torch.from_numpy(t).double()).square().mean()
        loss.backward()
        return dict(y=h.detach(), gradients=torch.cat([v.grad.ravel() for v in p]),
                    loss=float(loss.detach()))
    batch = case["kind"] == "batch"
    problems = _problems(case, seed) if batch else [_problem(case, seed)]
    x, y, rc, obj, rel, restarts = _pdhg(_Lps(problems), case)
    out = dict(primal=x, dual=y, reduced_costs=rc)
    if batch:
        out["objective"] = obj
    else:
        out["objective"] = float(obj[0])
        if case["precision"] != "mixed":
            out["relative_kkt"] = float(rel[0])
    return out
