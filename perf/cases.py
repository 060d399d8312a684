"""Timed workloads of the engine, each through a public entry point.

The listed cases are what programs have this engine do: linear programs from a
branch-and-bound node (a hundred columns) to 40M nonzeros, in both forms (FP64,
FP32 with FP64 refinement), from host arrays and from device-resident models,
cold and from a starting point; batches of uneven LPs; the node LPs of a
branching round; a training step's gradient of the learned warm start.  Solves run a fixed iteration budget
at a tolerance they do not reach within it, as a solver under a limit does, so
that a case is the same work for every seed.

``draw`` gives further cases of the same ranges; ``exact`` restates the PDHG
method and the network in plain FP64 torch.
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.abspath("markov-zip1_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import mcpdlp  # noqa: E402
from mcpdlp import learn  # noqa: E402

TOL = 1e-8


# --------------------------------------------------------------------- cases
def _solve(name, family, m, n, k, precision, memory, iterations, warm=False):
    c = {"op": "solve", "family": family, "m": m, "n": n, "k": k, "precision": precision,
         "memory": memory, "iterations": iterations, "warm": warm}
    return {"name": name, **c} if name else c


def listed():
    return [
        # the relaxation of one branch-and-bound node: the smallest call, all latency
        _solve("node_lp", "random", 61, 149, 4, "fp64", "host", 200),
        # the small LP with known optimum (1000 x 3000, 18k nonzeros), default options
        _solve("small_lp", "random", 1000, 3000, 6, "fp64", "host", 400),
        # transportation LP, 173 suppliers and 307 customers: two entries per column, rows of hundreds;
        # the budget ends inside a restart period
        _solve("transport", "transport", 173, 307, 2, "fp64", "host", 410),
        # a changed model solved again from the previous solution (warm start)
        _solve("resolve", "random", 4001, 12_007, 9, "fp64", "host", 400, warm=True),
        # a model as read from a file, odd sizes, in the mixed form
        _solve("medium_fp32", "random", 20011, 50021, 8, "fp32_refine", "host", 400),
        # 4M nonzeros: 1/10 of the large LP in every dimension
        _solve("large_fp64", "random", 200_000, 500_000, 8, "fp64", "device", 400),
        # wide-ranging magnitudes (1e-3..1e3), some columns boxed, 9M nonzeros
        _solve("precision_fp32", "precision", 300_007, 900_001, 10, "fp32_refine", "device", 400),
        # the headline LP, 2M x 5M with 40M nonzeros, in both forms
        _solve("headline_fp64", "random", 2_000_000, 5_000_000, 8, "fp64", "device", 800),
        _solve("headline_fp32", "random", 2_000_000, 5_000_000, 8, "fp32_refine", "device", 800),
        # independent LPs of uneven size solved together
        {"name": "batch", "op": "batch", "count": 48, "m_lo": 100, "m_hi": 4000, "precision": "fp64",
         "iterations": 400},
        # a branching round: node LPs that differ from their parent in a few bounds
        {"name": "node_round", "op": "variants", "m": 2000, "n": 6000, "k": 8, "count": 128,
         "precision": "fp32_refine", "iterations": 400},
        # forward and backward of the learned warm start on one training instance
        {"name": "learn_grad", "op": "grad", "m": 3000, "n": 9001, "k": 6},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    u = rng.random()
    precision = "fp64" if rng.random() < 0.5 else "fp32_refine"
    if u < 0.10:
        s, d = _log_int(rng, 20, 500), _log_int(rng, 20, 500)
        return _solve(None, "transport", s, d, 2, precision, "host", rng.randint(150, 600))
    if u < 0.66:
        nnz = _log_int(rng, 500, 36_000_000)
        k = rng.randint(3, 12)
        n = max(nnz // k, 40)
        m = max(int(n * rng.uniform(0.25, 0.6)), k + 4)
        iters = rng.randint(150, 800)
        if nnz > 8_000_000:  # at most the headline's work
            iters = max(150, min(iters, int(24_000_000_000 / nnz)))
        return _solve(None, "precision" if rng.random() < 0.25 else "random", m, n, k, precision,
                      "host" if nnz < 2_000_000 else "device", iters, rng.random() < 0.2)
    if u < 0.78:
        lo = _log_int(rng, 50, 400)
        return {"op": "batch", "count": rng.randint(8, 64), "m_lo": lo, "m_hi": lo * rng.randint(4, 12),
                "precision": "fp64", "iterations": rng.randint(120, 400)}
    if u < 0.90:
        m = _log_int(rng, 200, 4000)
        return {"op": "variants", "m": m, "n": int(m * rng.uniform(2, 4)), "k": rng.randint(4, 10),
                "count": rng.randint(20, 160), "precision": precision, "iterations": rng.randint(120, 400)}
    m = _log_int(rng, 100, 20_000)
    return {"op": "grad", "m": m, "n": int(m * rng.uniform(2, 4)), "k": rng.randint(4, 8)}


# -------------------------------------------------------------------- inputs
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gen(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    return g


def _q(t, bits):
    """Rounded to a multiple of 2^-bits: products and sums below are then exact
    in any order, so a seed gives the same model every time."""
    return torch.round(t * 2.0 ** bits) / 2.0 ** bits


def _random_lp(seed, m, n, k, family="random"):
    """Equality rows, k entries per column at uniform-random distinct rows,
    with a known optimum: b = A x*, c = A'y* + s (s the reduced costs)."""
    g, dev = _gen(seed), _device()

    def rand(*shape):
        return torch.rand(*shape, generator=g, device=dev, dtype=torch.float64)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device=dev, dtype=torch.float64)

    rows = torch.sort((rand(n, k) * m).long().clamp_(max=m - 1), dim=1).values
    for t in range(1, k):  # distinct: push equal neighbours up, then back below m
        rows[:, t] = torch.maximum(rows[:, t], rows[:, t - 1] + 1)
    for t in range(k - 1, -1, -1):
        rows[:, t].clamp_(max=m - k + t)
    val = normal(n, k) if family == "random" else 10.0 ** (6.0 * rand(n, k) - 3.0) * torch.where(
        rand(n, k) < 0.5, -1.0, 1.0)
    val = _q(val, 20)
    val[val == 0] = 2.0 ** -20
    y = normal(m)
    interior = rand(n) < 0.7
    x = torch.where(interior, _q(0.1 + 4.9 * rand(n), 10), 0.0)
    s = torch.where(interior, 0.0, 0.1 + 1.9 * rand(n))
    hi = torch.full((n,), 10.0, dtype=torch.float64, device=dev)
    if family == "precision":
        box = 1.0 + 99.0 * rand(n)
        boxed = rand(n) < 0.2
        hi = torch.where(boxed, torch.maximum(box, x), math.inf)
    b = torch.zeros(m, dtype=torch.float64, device=dev)
    b.index_add_(0, rows.reshape(-1), (val * x[:, None]).reshape(-1))
    c = (val * y[rows]).sum(1) + s
    def np_(t):
        return t.cpu().numpy()
    return mcpdlp.Model(m, n, np.arange(n + 1, dtype=np.int64) * k, np_(rows.reshape(-1).int()),
                        np_(val.reshape(-1)), np_(c), np.zeros(n), np_(hi), np_(b), np_(b),
                        info={"x_star": np_(x), "y_star": np_(y)})


def _transport_lp(seed, S, D):
    """Supplies <=, demands =, Euclidean costs (points in the unit square)."""
    r = np.random.default_rng(seed)
    ps_, pd = r.random((S, 2)), r.random((D, 2))
    sup = r.exponential(size=S)
    dem = r.exponential(size=D)
    sup, dem = sup / sup.sum() * 1100.0, dem / dem.sum() * 1000.0
    cost = np.sqrt(((ps_[:, None] - pd[None]) ** 2).sum(-1)) * (1 + 0.1 * r.normal(size=(S, D)))
    rows = np.empty((S, D, 2), np.int32)
    rows[..., 0] = np.arange(S)[:, None]
    rows[..., 1] = S + np.arange(D)[None]
    n = S * D
    return mcpdlp.Model(S + D, n, np.arange(n + 1) * 2, rows.reshape(-1), np.ones(2 * n),
                        np.maximum(cost, 0.0).reshape(-1), np.zeros(n), np.full(n, np.inf),
                        np.concatenate([np.full(S, -np.inf), dem]), np.concatenate([sup, dem]))


def _model(case, seed):
    if case["family"] == "transport":
        return _transport_lp(seed, case["m"], case["n"])
    return _random_lp(seed, case["m"], case["n"], case["k"], case["family"])


def _batch_models(case, seed):
    r = np.random.default_rng(seed)
    out = []
    for b in range(case["count"]):
        # the shapes of the batch belong to the case, so that every seed is the same work
        rs = np.random.default_rng(1000 * case["m_lo"] + b)
        m = int(rs.integers(case["m_lo"], case["m_hi"] + 1))
        out.append(_random_lp(int(r.integers(1 << 40)), m, int(rs.integers(2 * m, 4 * m + 1)),
                              int(rs.integers(4, 13))))
    return out


def _node_bounds(model, count, seed):
    """Children of a parent: 1-10 columns each moved to floor or ceil around
    x*; a child whose bounds would cross is not created (that bound stays)."""
    r = np.random.default_rng(seed)
    x = model.info["x_star"]
    los, his = [], []
    for _ in range(count):
        lo, hi = model.var_lower.copy(), model.var_upper.copy()
        for j in r.choice(model.num_cols, size=min(int(r.integers(1, 11)), model.num_cols), replace=False):
            if r.random() < 0.5:
                hi[j] = max(math.floor(x[j]), lo[j])
            else:
                lo[j] = min(math.ceil(x[j]), hi[j])
        los.append(lo)
        his.append(hi)
    return los, his


def _options(case):
    o = mcpdlp.PdlpOptions(max_iterations=case["iterations"], precision=mcpdlp.Precision[case["precision"]])
    o.set_tolerance(TOL)
    return o


def _start(model, seed):
    """A starting point near the optimum, as the solution of the model before
    a change is."""
    r = np.random.default_rng(seed)
    x, y = model.info["x_star"], model.info["y_star"]
    return x + 0.05 * r.normal(size=len(x)), y + 0.05 * r.normal(size=len(y))


def prepare(case, seed):
    op = case["op"]
    if op == "grad":
        model = _random_lp(seed, case["m"], case["n"], case["k"])
        return {"op": op, "net": learn.WarmStartNet(0, seed=1),
                "target": learn.Target(model, model.info["x_star"], model.info["y_star"], 0.7)}
    st = {"op": op, "ctx": mcpdlp.Context(0)}
    st["options"] = _options(case)
    if op == "batch":
        st["models"] = _batch_models(case, seed)
    elif op == "variants":
        st["model"] = _random_lp(seed, case["m"], case["n"], case["k"])
        st["lo"], st["hi"] = _node_bounds(st["model"], case["count"], seed)
    else:
        model = _model(case, seed)
        x0, y0 = _start(model, seed) if case["warm"] else (None, None)
        if case["memory"] == "device":
            if x0 is not None:
                x0, y0 = torch.from_numpy(x0).cuda(), torch.from_numpy(y0).cuda()
            st["model"] = mcpdlp.DeviceModel(model)
            st["x"] = torch.zeros(model.num_cols, dtype=torch.float64, device="cuda")
            st["y"] = torch.zeros(model.num_rows, dtype=torch.float64, device="cuda")
        else:
            st["model"] = model
        st["options"].initial_primal, st["options"].initial_dual = x0, y0
    return st


# ---------------------------------------------------------------------- runs
def _result(r):
    return {"primal": r.primal, "dual": r.dual, "objective": r.objective, "iterations": r.iterations,
            "status": int(r.status)}


def _results(rs):
    return {"primal": np.concatenate([r.primal for r in rs]), "dual": np.concatenate([r.dual for r in rs]),
            "objective": np.array([r.objective for r in rs]),
            "iterations": np.array([r.iterations for r in rs], np.int64),
            "status": np.array([int(r.status) for r in rs], np.int64)}


def run(state):
    op = state["op"]
    if op == "solve":
        if "x" in state:
            return _result(state["ctx"].solve_device(state["model"], state["options"], state["x"], state["y"]))
        return _result(state["ctx"].solve(state["model"], state["options"]))
    if op == "batch":
        return _results(state["ctx"].solve_batch(state["models"], state["options"]))
    if op == "variants":
        return _results(state["ctx"].solve_variants(state["model"], state["lo"], state["hi"], state["options"]))
    loss, grad = state["net"].loss_and_grad(state["target"])
    return {"loss": loss, "grad": grad}


# --------------------------------------------------------------------- work
def _iteration_bytes(nnz, m, n, precision):
    """Both matrix passes of one iteration and every vector it reads or writes."""
    if precision == "fp64":
        return 24 * nnz + 68 * m + 84 * n
    return 16 * nnz + 36 * m + 44 * n


def _sizes(case):
    if case.get("family") == "transport":
        S, D = case["m"], case["n"]
        return 2 * S * D, S + D, S * D
    return case["n"] * case["k"], case["m"], case["n"]


def work(case):
    op = case["op"]
    if op == "batch":
        nnz = m = n = 0
        for b in range(case["count"]):
            rs = np.random.default_rng(1000 * case["m_lo"] + b)
            mb = int(rs.integers(case["m_lo"], case["m_hi"] + 1))
            nb = int(rs.integers(2 * mb, 4 * mb + 1))
            nnz, m, n = nnz + nb * int(rs.integers(4, 13)), m + mb, n + nb
    else:
        nnz, m, n = _sizes(case)
    model = 12 * nnz + 28 * n + 16 * m  # read once
    if op == "grad":
        layer = (n + m) * 2 * 2 * 64 * 64 + 2 * 2 * nnz * 64
        return {"bytes": model + 3 * (n + m) * 64 * 4 * 4 * 2, "flops": 3 * 3 * layer}
    its = case["iterations"]
    if op == "variants":
        K = case["count"]
        v = 8 if case["precision"] == "fp64" else 4
        per = 24 * nnz + K * v * (8 * n + 6 * m)  # the matrix once for all variants
        return {"bytes": model + K * 8 * (2 * n + n + m) + its * per, "flops": its * K * (4 * nnz + 12 * (m + n))}
    return {"bytes": model + 8 * (n + m) + its * _iteration_bytes(nnz, m, n, case["precision"]),
            "flops": its * (4 * nnz + 12 * (m + n))}


# -------------------------------------------------------------------- exact
def _pdlp64(model, iterations, lo=None, hi=None, start=None):
    """Restarted PDHG in FP64, from the cold point or from `start`: Ruiz (10 passes), adaptive
    step size and primal weight, a restart check every 40 iterations."""
    dev = _device()

    def t(a):
        return torch.as_tensor(np.asarray(a), device=dev).double()

    m, n = model.num_rows, model.num_cols
    cs = torch.as_tensor(model.col_start, device=dev).long()
    ri = torch.as_tensor(model.row_index, device=dev).long()
    col = torch.repeat_interleave(torch.arange(n, device=dev), cs[1:] - cs[:-1])
    v = t(model.value).clone()
    lo0, hi0 = t(model.var_lower if lo is None else lo), t(model.var_upper if hi is None else hi)
    bl0, bh0, obj = t(model.row_lower), t(model.row_upper), t(model.objective)
    dr = torch.ones(m, dtype=torch.float64, device=dev)
    dc = torch.ones(n, dtype=torch.float64, device=dev)

    def line_max(index, size):
        z = torch.zeros(size, dtype=torch.float64, device=dev).scatter_reduce_(0, index, v.abs(), "amax")
        return torch.where(z == 0, 1.0, z)

    for _ in range(10):
        rm, cm = line_max(ri, m), line_max(col, n)
        if float((1 - rm).abs().max()) < 1e-3 and float((1 - cm).abs().max()) < 1e-3:
            break
        er, ec = 1 / rm.sqrt(), 1 / cm.sqrt()
        v *= er[ri] * ec[col]
        dr *= er
        dc *= ec
    big = 1e300
    lo_, hi_, bl, bh = lo0 / dc, hi0 / dc, bl0 * dr, bh0 * dr
    lo_, bl = lo_.clamp(min=-big), bl.clamp(min=-big)
    hi_, bh = hi_.clamp(max=big), bh.clamp(max=big)
    c = obj * dc
    order = torch.argsort(ri * n + col)
    rs = torch.zeros(m + 1, dtype=torch.long, device=dev)
    rs[1:] = torch.cumsum(torch.bincount(ri, minlength=m), 0)
    A = torch.sparse_csr_tensor(rs, col[order], v[order], size=(m, n))
    At = torch.sparse_csr_tensor(cs, ri, v, size=(n, m))
    ones_n = torch.ones(n, dtype=torch.float64, device=dev)
    ones_m = torch.ones(m, dtype=torch.float64, device=dev)
    cn = torch.sparse_csr_tensor(cs, ri, v.abs(), size=(n, m)) @ ones_m
    rn = torch.sparse_csr_tensor(rs, col[order], v[order].abs(), size=(m, n)) @ ones_n
    cn, rn = torch.where(cn < 1e-12, 1.0, cn), torch.where(rn < 1e-12, 1.0, rn)
    fin = torch.cat([bl, bh])
    fin = fin[fin.abs() < 1e299].abs()
    c_norm, b_norm = max(1.0, float(c.abs().max())), max(1.0, float(fin.max()) if len(fin) else 0.0)
    c_scale = max(1.0, float(obj.abs().max()))
    omega = min(max(math.sqrt(c_norm / b_norm), 0.01), 100.0)
    eta, last, count, since = 0.9, 1e300, 0, 0
    x = torch.zeros(n, dtype=torch.float64, device=dev) if start is None else t(start[0]) / dc
    y = torch.zeros(m, dtype=torch.float64, device=dev) if start is None else t(start[1]) / dr
    x = x.clamp(lo_, hi_)
    xa, ya = x.clone(), y.clone()

    def residuals():
        xu, yu = xa * dc, ya * dr
        ax, g = (A @ xa) / dr, obj + (At @ ya) / dc

        def violation(a, l, h):
            p = a.clamp(l, h)
            return float(((a - p).abs() / (1 + torch.maximum(a.abs(), p.abs()))).max())
        primal = max(violation(ax, bl0, bh0), violation(xu, lo0, hi0))
        dual = float((xu - (xu - g).clamp(lo0, hi0)).norm()) / c_scale
        pobj = float((obj * xu).sum())
        bound = torch.where(g > 0, lo0, torch.where(g < 0, hi0, 0.0))
        rb = torch.where(yu > 0, bh0, torch.where(yu < 0, bl0, 0.0))
        dobj = float(torch.where(bound.isfinite(), g * bound, 0.0).sum()) - float(
            torch.where(rb.isfinite(), yu * rb, 0.0).sum())
        gap = abs(pobj - dobj) / (1 + abs(pobj) + abs(dobj))
        return primal, dual, gap, pobj

    it, pobj, status = 0, 0.0, 1
    while it < iterations:
        span = min(40, iterations - it)
        for k in range(span):
            xn = (x - eta / omega / cn * (c + At @ y)).clamp(lo_, hi_)
            xbar = 2 * xn - x
            if (it + k) % 10 == 0:
                d = xn - x
                d2, a2 = float((cn * d * d).sum()), float(((A @ d) ** 2 / rn).sum())
                if d2 > 1e-14 and a2 > 1e-14 and math.sqrt(a2 / d2) > 1e-6:
                    target = 0.95 / math.sqrt(a2 / d2)
                    if target < eta:
                        eta = max(0.1, target, eta * 0.8)
                    elif target > 1.05 * eta and eta < 0.99:
                        eta = min(0.99, eta * 1.05)
            sigma = eta * omega / rn
            w = y + sigma * (A @ xbar)
            y = w - sigma * (w / sigma).clamp(bl, bh)
            x = xn
            xa += (x - xa) / (count + k + 1)
            ya += (y - ya) / (count + k + 1)
        it += span
        primal, dual, gap, pobj = residuals()
        if span < 40:
            break
        if max(primal, dual, gap) <= TOL:
            status = 0
            break
        score = max(primal, dual, gap)
        since += span
        if score <= 0.368 * last or (since >= 200 and score < last):
            if primal > 1e-12 and dual > 1e-12:
                omega = min(max(omega * math.sqrt(min(max(math.sqrt(primal / dual), 0.05), 20.0)), 1e-6), 1e6)
            x, y, count, since, last = xa.clone(), ya.clone(), 0, 0, score
        else:
            count += span
    return {"primal": (xa * dc).cpu().numpy(), "dual": (ya * dr).cpu().numpy(), "objective": pobj,
            "iterations": it, "status": status}


def _grad64(target, params):
    """The network of the learned warm start in FP64: bipartite message
    passing (hidden width 64, 3 rounds) and its squared-error loss."""
    H, md = 64, target.model
    m, n = md.num_rows, md.num_cols
    p = torch.tensor(params, dtype=torch.float64, requires_grad=True)
    at = 0

    def take(*shape):
        nonlocal at
        size = int(np.prod(shape))
        at += size
        return p[at - size:at].reshape(shape)

    wve, bve, wce, bce = take(6, H), take(H), take(5, H), take(H)
    layers = [[take(H, H), take(H, H), take(H), take(H, H), take(H, H), take(H)] for _ in range(3)]
    wx, bx, wy, by, uv, uc, bw = take(H), take(1), take(H), take(1), take(H), take(H), take(1)

    def t(a):
        return torch.as_tensor(np.asarray(a)).double()

    ri = torch.as_tensor(md.row_index).long()
    col = torch.repeat_interleave(torch.arange(n), torch.as_tensor(np.diff(md.col_start)).long())
    v = t(md.value.astype(np.float32))
    rn = torch.zeros(m, dtype=torch.float64).index_add_(0, ri, v.abs())
    cn = torch.zeros(n, dtype=torch.float64).index_add_(0, col, v.abs())
    bs = max(1.0, float(np.abs(md.row_upper).max()))
    cscale = max(1.0, float(np.abs(md.objective).max()))
    lo, hi, b = t(md.var_lower), t(md.var_upper), t(md.row_lower)
    one = torch.ones(n, dtype=torch.float64)
    fv = torch.stack([t(md.objective) / cscale, one, one, (lo / bs).clamp(-10, 10), (hi / bs).clamp(-10, 10),
                      cn / cn.max()], 1)
    one = torch.ones(m, dtype=torch.float64)
    fc = torch.stack([b / bs, b / bs, one, one, rn / rn.max()], 1)
    vr = torch.where(rn > 0, 1 / rn, 0.0)[ri] * v
    vc = torch.where(cn > 0, 1 / cn, 0.0)[col] * v
    a_row = torch.sparse_coo_tensor(torch.stack([ri, col]), vr, (m, n)).coalesce()
    a_col = torch.sparse_coo_tensor(torch.stack([col, ri]), vc, (n, m)).coalesce()
    hv, hc = torch.relu(fv @ wve + bve), torch.relu(fc @ wce + bce)
    for wcs, wcn, bc, wvs, wvn, bv in layers:
        hc = torch.relu(hc @ wcs + torch.sparse.mm(a_row, hv) @ wcn + bc)
        hv = torch.relu(hv @ wvs + torch.sparse.mm(a_col, hc) @ wvn + bv)
    px, py = hv @ wx + bx, hc @ wy + by
    lw = hv.mean(0) @ uv + hc.mean(0) @ uc + bw
    loss = ((px - t(target.x) / bs) ** 2).mean() + ((py - t(target.y) / cscale) ** 2).mean() + \
        0.1 * ((lw - target.log_omega) ** 2).sum()
    loss.backward()
    return {"loss": float(loss), "grad": p.grad.numpy()}


def exact(case, seed):
    op = case["op"]
    if op == "grad":
        model = _random_lp(seed, case["m"], case["n"], case["k"])
        net = learn.WarmStartNet(0, seed=1)
        return _grad64(learn.Target(model, model.info["x_star"], model.info["y_star"], 0.7),
                       net.params.astype(np.float64))
    its = case["iterations"]
    if op == "solve":
        model = _model(case, seed)
        return _pdlp64(model, its, start=_start(model, seed) if case["warm"] else None)
    if case["count"] * its > 60_000:  # over 20 seconds, one LP after another
        return None
    if op == "batch":
        rs = [_pdlp64(m, its) for m in _batch_models(case, seed)]
    else:
        model = _random_lp(seed, case["m"], case["n"], case["k"])
        rs = [_pdlp64(model, its, lo, hi) for lo, hi in zip(*_node_bounds(model, case["count"], seed))]
    return {"primal": np.concatenate([r["primal"] for r in rs]), "dual": np.concatenate([r["dual"] for r in rs]),
            "objective": np.array([r["objective"] for r in rs]),
            "iterations": np.array([r["iterations"] for r in rs], np.int64),
            "status": np.array([r["status"] for r in rs], np.int64)}
