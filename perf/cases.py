"""Performance cases of the LIBOR-market-model pricing library.

Each case is one pass of work that a program using this library asks for,
through ``useful_code_b200.pricer.Pipeline``: whole two-pass Bermudan prices,
the first pass alone, a regression, nested regressions, pathwise Greeks, an
Andersen-Broadie bound and the plain staged chain, on the models of
``useful_code_b200.configs`` (c1: 20 rates, 3 factors; c2: 40 rates, 5
factors; c3 / c4: 80 rates, 10 factors; c5: 120 rates, 15 factors).

``exact`` restates every path in 64-bit torch, without the library: the Sobol
points from the direction integers, the exact inverse normal, the Brownian
bridge, the predictor-corrector evolution with the drift as a matrix product,
the products, the backward regression (nested too), and the Greeks by
automatic differentiation.
"""
from __future__ import annotations

import functools
import math
from dataclasses import replace

import numpy as np
import torch

from useful_code_b200 import market as mk
from useful_code_b200.pricer import LSInputs, LSResult, Pipeline, Selector

DEV = "cuda"
CHUNK = 1 << 17  # paths per 64-bit evaluation
RULE_PATHS = 1 << 13  # paths behind a frozen rule that a case starts from


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: a European caplet strip plus payer swap on the
        # small model at its stated path count (a pricing inside a quote loop)
        {"name": "strip_c1", "kind": "strip", "model": "c1", "n": 20, "paths": 16384,
         "offset": 0},
        # a quick Bermudan indication: few paths, odd counts, launch-bound
        {"name": "price_c2_quick", "kind": "price", "model": "c2", "n": 40, "reg": 4099,
         "paths": 10007},
        # the ordinary Bermudan valuation at its stated size
        {"name": "price_c2", "kind": "price", "model": "c2", "n": 40, "reg": 65536,
         "paths": 262144},
        # the headline valuation: 2^20 regression and 2^20 pricing paths
        {"name": "price_c3", "kind": "price", "model": "c3", "n": 80, "reg": 1 << 20,
         "paths": 1 << 20},
        # the largest model, a cancellable swap, ragged path counts
        {"name": "price_c5", "kind": "price", "model": "c5", "n": 120, "reg": 150001,
         "paths": 200003},
        # one shard of a regression run: the LS inputs of an odd path range
        {"name": "inputs_c3", "kind": "inputs", "model": "c3", "n": 80, "paths": 100003,
         "offset": 123457},
        # the regression alone on inputs already on the device
        {"name": "regress_c3", "kind": "regress", "model": "c3", "n": 80, "paths": 1 << 20},
        # the production setting: nested regressions of depth 4
        {"name": "nested_c3", "kind": "nested", "model": "c3", "n": 80, "reg": 1 << 18,
         "paths": 1 << 18, "depth": 4},
        # hedge ratios of the frozen-rule price: all deltas, dV/dA, vegas
        {"name": "greeks_c3", "kind": "greeks", "model": "c3", "n": 80, "paths": 1 << 18},
        # the same for the swaption-plus-cap portfolio on few paths
        {"name": "greeks_c4_small", "kind": "greeks", "model": "c4", "n": 80, "paths": 8192},
        # upper bound of the rule by nested simulation
        {"name": "bound_c3", "kind": "bound", "model": "c3", "n": 80, "outer": 96,
         "inner": 256},
        # the plain staged chain (the reference's kernels one by one)
        {"name": "staged_c2", "kind": "staged", "model": "c2", "n": 40, "reg": 32768,
         "paths": 65536},
    ]


SIZES = {"c1": 20, "c2": 40, "c3": 80, "c4": 80, "c5": 120, "t1": 20}


def draw(rng):
    kind = rng.choice(["strip", "price", "price", "price", "inputs", "regress", "nested",
                       "greeks", "greeks", "bound", "staged"])
    models = {"strip": ["c1"], "price": ["c2", "c3", "c4", "c5", "t1"],
              "inputs": ["c2", "c3", "c5"], "regress": ["c2", "c3", "c5"],
              "nested": ["c2", "c3"], "greeks": ["c1", "c3", "c4", "c5"],
              "bound": ["c2", "c3"], "staged": ["c1", "c2", "c3"]}
    model = rng.choice(models[kind])
    full = SIZES[model]
    n = rng.choice([full, rng.randint(full // 2, full)])

    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    # the most paths of this model that cost no more than the largest listed
    top = {"c1": 1 << 18, "c2": 1 << 19, "c3": 1 << 20, "c4": 1 << 19, "c5": 1 << 18,
           "t1": 1 << 18}[model]
    case = {"kind": kind, "model": model, "n": n}
    if kind == "strip":
        case.update(paths=log(1000, 1 << 17), offset=rng.randint(0, 1 << 20))
    elif kind == "price":
        case.update(reg=log(2000, top), paths=log(2000, top))
    elif kind == "inputs":
        case.update(paths=log(1000, top // 2), offset=rng.randint(0, 1 << 20))
    elif kind == "regress":
        case.update(paths=log(2000, top))
    elif kind == "nested":
        case.update(reg=log(1 << 14, top // 2), paths=log(4000, top // 2),
                    depth=rng.randint(2, 4))
    elif kind == "greeks":
        case.update(paths=4 * log(500, top // 16))
    elif kind == "bound":
        case.update(outer=rng.randint(10, 120), inner=128 * rng.randint(1, 4))
    else:
        case.update(reg=log(2000, top // 16), paths=log(2000, top // 8))
    return case


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
@functools.lru_cache(maxsize=32)
def _base_market(model, n):
    cfg = mk.make_config(model)
    if n != cfg.n:
        cfg = replace(cfg, n=n, f0=cfg.f0[:n].copy())
    return mk.build_market(cfg)


def _market(case, seed):
    """The model's market with today's curve (a seeded quadratic move of up to
    about 20 bp) and scrambler words of this seed."""
    base = _base_market(case["model"], case["n"])
    rng = np.random.default_rng([seed, 77])
    x = np.linspace(-1.0, 1.0, case["n"])
    c = rng.uniform(-0.001, 0.001, 3)
    f0 = (base.f0 + c[0] + c[1] * x + 0.5 * c[2] * x * x).astype(np.float32)
    words = rng.integers(0, 1 << 32, base.scramblers.size, dtype=np.uint32)
    return replace(base, cfg=replace(base.cfg, f0=f0), f0=f0, scramblers=words)


def _ls_inputs(m, P, offset):
    """LS inputs from the 64-bit model, as float32 device arrays."""
    vars_, ex, cf, num = _first_pass64(m, P, offset)
    return LSInputs(vars_.float(), ex.float(), cf.float(), num.float())


def _frozen_rule(m):
    """An exercise rule from an earlier calibration on a few paths."""
    vars_, ex, cf, num = _first_pass64(m, RULE_PATHS, 1 << 22)
    r = _regress64(m, vars_, ex, cf, num)
    return LSResult(r["beta"][:, 0].contiguous(), r["means"][:, 0].float().contiguous(),
                    r["sds"][:, 0].float().contiguous(), None,
                    torch.zeros(1, dtype=torch.int32, device=DEV),
                    torch.zeros(1, dtype=torch.float64, device=DEV))


def prepare(case, seed):
    m = _market(case, seed)
    s = {"case": case, "mkt": m, "pipe": Pipeline(m)}
    kind = case["kind"]
    if kind == "regress":
        s["ls"] = _ls_inputs(m, case["paths"], 0)
    elif kind in ("greeks", "bound"):
        s["rule"] = _frozen_rule(m) if len(m.ex_steps) else None
        s["seed"] = 20240601 + seed
    return s


def run(s):
    c, pipe = s["case"], s["pipe"]
    kind = c["kind"]
    if kind == "strip":
        return pipe.second_pass(c["paths"], c["offset"], None)
    if kind == "price":
        return pipe.price(c["reg"], c["paths"])
    if kind == "staged":
        return pipe.price(c["reg"], c["paths"], mode="staged", batch=32768)
    if kind == "nested":
        return pipe.price(c["reg"], c["paths"], select=Selector.production(c["depth"]))
    if kind == "inputs":
        ls = pipe.first_pass(c["paths"], c["offset"])
        return {"vars": ls.vars, "ex": ls.ex, "cf": ls.cf, "num": ls.num}
    if kind == "regress":
        r = pipe.regress(s["ls"])
        return {"beta": r.beta, "means": r.means, "sds": r.sds, "price": r.price,
                "status": r.status}
    if kind == "greeks":
        g = pipe.greeks(c["paths"], 0, s["rule"])
        return {"price": g.price, "delta": g.delta, "abar": g.abar, "vega": g.vega_rate,
                "step": g.exercise_step}
    b = pipe.andersen_broadie(s["rule"], c["outer"], 1 << 16, c["inner"], s["seed"], keep=True)
    return {"lower": b.lower, "lower_se": b.lower_se, "gap": b.gap, "gap_se": b.gap_se,
            "Q": b.Q, "Z": b.Z, "X": b.X}


# --------------------------------------------------------------------------
# work and tolerance
# --------------------------------------------------------------------------
def _path_flops(n, F):
    # per (rate, step): two products with the factor vectors and two updates
    # of them, and 12 scalar operations; per (step, factor): the inverse
    # normal's two polynomials and three operations of the bridge
    return n * (n + 1) // 2 * (8 * F + 12) + n * F * 30


def work(case):
    kind, n = case["kind"], case["n"]
    F = _base_market(case["model"], n).cfg.F
    E = 0 if case["model"] in ("c1", "t1") else n
    nb = {"c2": 6, "c5": 12}.get(case["model"], 10)
    model_bytes = 4 * (n * n * F + n * n + 33 * n * F)
    gram = (nb + 1) * (nb + 2) + 4 * nb  # per path and date, with the decision
    one = _path_flops(n, F)
    if kind == "strip":
        return {"bytes": model_bytes + 4 * case["paths"], "flops": one * case["paths"]}
    if kind == "inputs":
        return {"bytes": model_bytes + 24 * E * case["paths"], "flops": one * case["paths"]}
    if kind == "regress":
        return {"bytes": 24 * E * case["paths"], "flops": gram * E * case["paths"]}
    if kind in ("price", "staged", "nested"):
        reg = case["reg"] if E else 0
        return {"bytes": model_bytes + 8,
                "flops": one * (reg + case["paths"]) + gram * E * reg * case.get("depth", 1)}
    if kind == "greeks":
        # the adjoint: four products with the factor vectors and the path's
        # row of dV/dA (two more) per rate and step
        back = n * (n + 1) // 2 * 12 * F
        return {"bytes": model_bytes + 8 * n * n * F + 4 * case["paths"],
                "flops": (one + back) * case["paths"]}
    inner = case["outer"] * case["inner"]
    steps = sum((n - e - 1) * (n - e) // 2 * (8 * F + 12) + (n - e - 1) * F * 75
                for e in range(E - 1))
    return {"bytes": model_bytes + 20 * E * case["outer"],
            "flops": one * case["outer"] + inner * steps}


def tolerance(case):
    """About four times the largest distance from ``exact`` measured over the
    listed and some drawn cases.  Where exercise decisions enter, a path whose
    exercise value equals its estimate to rounding may decide the other way:
    on a few thousand paths one such path moves a price by a few 1e-4, and
    nested regressions, fitted to the paths nearest the boundary, move by
    about 2e-3.  A caplet kink does the same to one path's derivative."""
    return {
        "strip": {"rel": 2e-6},
        "inputs": {"rel": 2e-5},
        "price": {"rel": 1e-3},
        "staged": {"rel": 1e-3},
        "nested": {"rel": 8e-3},
        "regress": {"rel": 1e-3},
        "greeks": {"rel": 2e-3, "differ": 1e-3},
        "bound": {"rel": 3e-3, "differ": 1e-3},
    }[case["kind"]]


# --------------------------------------------------------------------------
# the same in 64 bits
# --------------------------------------------------------------------------
def _tables(n, F):
    """Bridge stages (target, left, right, weights) and the diagonal
    allocation of Sobol dimensions [factor][stage]."""
    stages, built = [(n - 1, -1, -1, 0.0, 0.0, math.sqrt(n))], [False] * n
    built[n - 1] = True
    j = 0
    for _ in range(1, n):
        while built[j]:
            j += 1
        k = j
        while not built[k]:
            k += 1
        mid = j + ((k - 1 - j) >> 1)
        built[mid] = True
        t0, tm, tk = float(j), mid + 1.0, k + 1.0  # t0 = time of point j - 1
        stages.append((mid, j - 1, k, (tk - tm) / (tk - t0), (tm - t0) / (tk - t0),
                       math.sqrt((tm - t0) * (tk - tm) / (tk - t0))))
        j = k + 1
        if j >= n:
            j = 0
    alloc = np.zeros((F, n), np.int64)
    count = 0
    for d in range(F + n - 1):  # anti-diagonals, from the last factor upwards
        for i in range(min(d, F - 1), -1, -1):
            if d - i < n:
                alloc[i, d - i] = count
                count += 1
    return stages, alloc


def _normals64(m, P, offset):
    """Bridged increments [steps][factors][P]."""
    n, F = m.cfg.n, m.cfg.F
    stages, alloc = _tables(n, F)
    dirs = torch.from_numpy(m.directions.astype(np.int64)).to(DEV)
    scr = torch.from_numpy(m.scramblers.astype(np.int64)).to(DEV)
    idx = torch.arange(1 + offset, 1 + offset + P, device=DEV, dtype=torch.int64)
    gray = idx ^ (idx >> 1)
    bits = int(1 + offset + P).bit_length()
    out = torch.empty(n, F, P, dtype=torch.float64, device=DEV)
    for f in range(F):
        d = torch.from_numpy(alloc[f]).to(DEV)
        x = torch.zeros(n, P, dtype=torch.int64, device=DEV)
        for b in range(bits):
            x ^= dirs[d, b][:, None] * ((gray >> b) & 1)[None]
        x ^= torch.where(d < m.scramble_dims, scr[d], torch.zeros_like(d))[:, None]
        u = torch.minimum(x, (1 << 32) - x).clamp(min=1).double() * 2.0 ** -32
        z = torch.special.ndtri(u)
        z = torch.where(x >= 1 << 31, -z, z)
        w = out[:, f]
        for i, (t, lo, hi, lw, rw, sd) in enumerate(stages):
            y = sd * z[i]
            if hi >= 0:
                y = y + rw * w[hi]
            if lo >= 0:
                y = y + lw * w[lo]
            w[t] = y
        w[1:] = w[1:] - w[:-1].clone()
    return out


def _evolve64(m, lf, z, A, s0=0, N=None):
    """Steps s0.. of the predictor-corrector evolution; yields (s, N, f, P)
    after each: the numeraire at T_s, the forwards s.. and the discount
    factors P(T_s, T_{r+1})."""
    n, tau, d = m.cfg.n, float(m.taus[0]), float(m.disp[0])
    N = torch.ones_like(lf[0]) if N is None else N
    first = None

    def drift_factor(x):
        F = torch.exp(x)
        return F * tau / (1.0 + tau * (F - d))

    for s in range(s0, n):
        if first is not None:
            N = N * (1.0 + tau * first)
        a, x = A[s, s:], lf[s - n:]
        C = torch.tril(a @ a.T)
        g = drift_factor(x)
        x = x + C @ g + a @ z(s) - 0.5 * (a * a).sum(1, keepdim=True)
        x = x + 0.5 * (C @ (drift_factor(x) - g))
        lf = torch.clamp(x, max=m.cfg.cutoff)
        f = torch.exp(lf) - d
        first = f[0]
        yield s, N, f, torch.cumprod(1.0 / (1.0 + tau * f), 0), lf


def _start64(m, P):
    A = torch.from_numpy(m.A).to(DEV).double()
    lf0 = torch.log(torch.from_numpy(m.f0).to(DEV).double() + float(m.disp[0]))
    return A, lf0[:, None].expand(m.cfg.n, P)


def _date64(m, s, f, P):
    """Basis variables, exercise value and coupon of the date at T_s."""
    cfg, tau = m.cfg, float(m.taus[0])
    ann, Pn = tau * P.sum(0), P[-1]
    if cfg.product in ("swaption", "bermudan_cap"):
        sr = (1.0 - Pn) / ann
        return (f[0], sr, ann, torch.clamp((sr - cfg.strike) * ann, min=0.0),
                torch.zeros_like(ann))
    sr = (P[0] - Pn) / (ann - tau * P[0]) if s + 1 < cfg.n else (1.0 - Pn) / ann
    return (f[0], sr, tau * Pn, torch.zeros_like(ann),
            tau * (f[0] - cfg.strike) * cfg.pay_receive * P[0])


def _first_pass64(m, P, offset):
    E = len(m.ex_steps)
    vars_ = torch.empty(E, 3, P, dtype=torch.float64, device=DEV)
    ex, cf, num = (torch.empty(E, P, dtype=torch.float64, device=DEV) for _ in range(3))
    for c in range(0, P, CHUNK):
        b = min(CHUNK, P - c)
        z = _normals64(m, b, offset + c)
        A, lf = _start64(m, b)
        for s, N, f, D, _ in _evolve64(m, lf, lambda s: z[s], A):
            v0, v1, v2, x, cpn = _date64(m, s, f, D)
            for k, v in enumerate((v0, v1, v2)):
                vars_[s, k, c:c + b] = v
            ex[s, c:c + b], cf[s, c:c + b], num[s, c:c + b] = x, cpn, N
    return vars_, ex, cf, num


def _phi64(m, e, x):
    """Basis functions [K][P] of the standardised variables x [3][P]."""
    rows = []
    for k in range(int(m.nbasis[e])):
        y = torch.ones_like(x[0])
        for v in range(3):
            if m.mono[e, k, v]:
                y = y * x[v] ** int(m.mono[e, k, v])
        rows.append(y)
    return torch.stack(rows)


def _estimate64(m, e, vars_e, ex_e, rule):
    """Continuation estimate by the rule's chain of regressions."""
    depth = rule["beta"].shape[1]
    K = int(m.nbasis[e])
    est = open_ = None
    for d in range(depth):
        x = (vars_e - rule["means"][e, d, :, None]) / rule["sds"][e, d, :, None]
        t = rule["beta"][e, d, :K] @ _phi64(m, e, x)
        est = t if est is None else torch.where(open_, t, est)
        if d + 1 == depth:
            break
        net = t - ex_e
        inside = (net > rule["cuts"][e, d, 0]) & (net < rule["cuts"][e, d, 1])
        open_ = inside if open_ is None else open_ & inside
    return est


def _select64(net, sel):
    """Half-width of the band of net values that keeps about a fraction of
    them (the fraction selector's search), and how many it keeps."""
    srt = torch.sort(net.abs()).values
    n = net.numel()

    def count(g):
        return int(torch.searchsorted(srt, torch.tensor([g], dtype=srt.dtype, device=DEV),
                                      right=True))

    lo_t, hi_t = int(n * sel.lower_frac), int(n * sel.upper_frac)
    if lo_t < n < hi_t:
        return 1e4, count(1e4)
    g = float((net.square().mean() - net.mean() ** 2).sqrt()) * sel.sds
    c, left = count(g), 500
    while c < lo_t and left:
        g, left = g / sel.multiplier, left - 1
        c = count(g)
    if c < hi_t:
        return g, c
    lo = g * sel.multiplier
    c = count(lo)
    while c > hi_t and left:
        lo, left = lo * sel.multiplier, left - 1
        c = count(lo)
    if c > lo_t:
        return lo, c
    hi = g
    g = 0.5 * (lo + hi)
    c = count(g)
    while (c < lo_t or c > hi_t) and hi - lo > 1e-6:
        lo, hi = (g, hi) if c < lo_t else (lo, g)
        g = 0.5 * (lo + hi)
        c = count(g)
    return g, c


def _regress64(m, vars_, ex, cf, num, sel=None):
    E, P = ex.shape
    D = sel.depth if sel else 1
    rule = {"beta": torch.zeros(E, D, 16, dtype=torch.float64, device=DEV),
            "means": torch.zeros(E, D, 3, dtype=torch.float64, device=DEV),
            "sds": torch.ones(E, D, 3, dtype=torch.float64, device=DEV),
            "cuts": torch.zeros(E, D, 2, dtype=torch.float64, device=DEV)}
    y = torch.zeros(P, dtype=torch.float64, device=DEV)
    for e in range(E - 1, -1, -1):
        K, ve, xe, ce = int(m.nbasis[e]), vars_[e].double(), ex[e].double(), cf[e].double()
        keep = None
        for d in range(D):
            vk, tk = (ve, ce + y) if keep is None else (ve[:, keep], (ce + y)[keep])
            mean = vk.mean(1)
            sd = ((vk * vk).mean(1) - mean * mean).clamp(min=0.0).sqrt()
            sd = torch.where(sd > 0, sd, torch.ones_like(sd))
            phi = _phi64(m, e, (vk - mean[:, None]) / sd[:, None])
            G, b = phi @ phi.T / vk.shape[1], phi @ tk / vk.shape[1]
            L, info = torch.linalg.cholesky_ex(G)
            if int(info) == 0:
                rule["beta"][e, d, :K] = torch.cholesky_solve(b[:, None], L)[:, 0]
            rule["means"][e, d], rule["sds"][e, d] = mean, sd
            if d + 1 == D:
                break
            net = rule["beta"][e, d, :K] @ phi - (xe if keep is None else xe[keep])
            if d == 0 and (float(net.max()) <= 0.0 or float(net.min()) >= 0.0):
                break
            c, after = _select64(net, sel)
            if after <= sel.min_paths:
                break
            rule["cuts"][e, d, 0], rule["cuts"][e, d, 1] = -c, c
            inside = net.abs() <= c
            if keep is None:
                keep = inside
            else:
                keep = keep.clone()
                keep[keep.clone()] = inside
        est = _estimate64(m, e, ve, xe, rule)
        y = torch.where(xe > est, xe, ce + y)
        if e > 0:
            y = y * num[e - 1].double() / num[e].double()
    rule["price"] = (y / num[0].double()).mean()
    return rule


def _payoffs64(m, P, offset, rule, A=None, lf=None, z=None):
    """Deflated payoffs [P] and exercise steps [P] under a frozen rule."""
    cfg, n, tau = m.cfg, m.cfg.n, float(m.taus[0])
    z = _normals64(m, P, offset) if z is None else z
    A0, lf0 = _start64(m, P)
    A, lf = (A0 if A is None else A), (lf0 if lf is None else lf)
    pay = torch.zeros(P, dtype=torch.float64, device=DEV)
    step = torch.full((P,), n, dtype=torch.int64, device=DEV)
    live = torch.ones(P, dtype=torch.bool, device=DEV)
    paid = torch.zeros(P, dtype=torch.float64, device=DEV)
    for s, N, f, D, _ in _evolve64(m, lf, lambda s: z[s], A):
        if cfg.product == "european":
            flow = torch.clamp(f[0] - cfg.cap_strike, min=0.0) + (f[0] - cfg.strike) * \
                cfg.pay_receive
            pay = pay + tau * flow * D[0] / N
            continue
        if cfg.product == "tarn":
            c = torch.clamp((cfg.strike - cfg.tarn_multiplier * f[0]) * tau, min=0.0)
            stop = (paid + c >= cfg.tarn_total) | (s + 1 == n)
            flow = tau * f[0] + torch.where(stop, paid - cfg.tarn_total, -c)
            pay = pay + torch.where(live, flow * D[0] / N, torch.zeros_like(pay))
            paid = torch.where(live & ~stop, paid + c, paid)
            live = live & ~stop
            continue
        if cfg.product == "bermudan_cap":
            pay = pay + tau * torch.clamp(f[0] - cfg.cap_strike, min=0.0) * D[0] / N
        v0, v1, v2, x, cpn = _date64(m, s, f, D)
        with torch.no_grad():
            est = _estimate64(m, s, torch.stack((v0, v1, v2)), x, rule)
            now = live & (x > est)
            step[now] = s
        zero = torch.zeros_like(pay)
        pay = pay + torch.where(now, x / N, zero) + torch.where(live & ~now, cpn / N, zero)
        live = live & ~now
    return pay, step


def _price64(case, m, sel):
    scale = 1.0 / (1.0 + float(m.f0[0]) * float(m.rate_times[0]))
    rule = out = None
    offset = case["reg"]
    if len(m.ex_steps):
        rule = _regress64(m, *_first_pass64(m, case["reg"], 0), sel)
        out = float(rule["price"]) * scale
    total = 0.0
    for c in range(0, case["paths"], CHUNK):
        b = min(CHUNK, case["paths"] - c)
        total += float(_payoffs64(m, b, offset + c, rule)[0].sum())
    price = {"price": torch.tensor(total / case["paths"] * scale, dtype=torch.float64)}
    return price if out is None else {
        **price, "insample": torch.tensor(out, dtype=torch.float64), "ls_status": None}


def _rule64(rule):
    if rule is None:
        return None
    return {"beta": rule.beta[:, None], "means": rule.means.double()[:, None],
            "sds": rule.sds.double()[:, None]}


def _greeks64(case, m, rule):
    n, P = m.cfg.n, case["paths"]
    A = torch.from_numpy(m.A).to(DEV).double().requires_grad_()
    f0 = torch.from_numpy(m.f0).to(DEV).double().requires_grad_()
    total, chunk = 0.0, min(P, 1 << 16)
    for c in range(0, P, chunk):
        b = min(chunk, P - c)
        with torch.no_grad():
            z = _normals64(m, b, c)
        lf = torch.log(f0 + float(m.disp[0]))[:, None].expand(n, b)
        pay, _ = _payoffs64(m, b, c, rule, A, lf, z)
        v = pay.sum() / P / (1.0 + f0[0] * float(m.rate_times[0]))
        v.backward()
        total += float(v.detach())
    vega = (A.grad * A.detach()).sum((0, 2))
    return {"price": torch.tensor(total, dtype=torch.float64), "delta": f0.grad,
            "abar": A.grad, "vega": vega, "step": None}


def _philox64(c, k0, k1):
    """Philox4x32-10 on int64 tensors holding 32-bit words."""
    def mul(a, x):  # 32 x 32 bits -> (high, low)
        lo, hi = (x & 0xFFFF) * a, (x >> 16) * a
        t = lo + ((hi & 0xFFFF) << 16)
        return (hi >> 16) + (t >> 32), t & 0xFFFFFFFF

    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
    return c


def _bound64(case, m, rule, seed):
    n, F, K, I = m.cfg.n, m.cfg.F, case["outer"], case["inner"]
    z = _normals64(m, K, 1 << 16)
    A, lf = _start64(m, K)
    X, Z = (torch.zeros(n, K, dtype=torch.float64, device=DEV) for _ in range(2))
    starts = []  # state at the start of step s + 1 = after step s
    for s, N, f, D, lfn in _evolve64(m, lf, lambda s: z[s], A):
        v0, v1, v2, x, _ = _date64(m, s, f, D)
        X[s] = (x > _estimate64(m, s, torch.stack((v0, v1, v2)), x, rule)).double()
        Z[s] = x / N
        starts.append((lfn[1:], N * (1.0 + float(m.taus[0]) * f[0])))
    Q = torch.zeros(n, K, dtype=torch.float64, device=DEV)
    p = torch.arange(K, device=DEV).repeat_interleave(I)
    i = torch.arange(I, device=DEV).repeat(K)
    # all inner paths of the dates before step s advance together: each date
    # joins at its own start
    def normals(s, e, pp, ii):
        rows = []
        for j in range((F + 3) // 4):
            w = _philox64([ii, pp, torch.full_like(pp, 4 * s + j), e],
                          seed & 0xFFFFFFFF, seed >> 32)
            rows += w
        x = torch.stack(rows[:F])
        u = torch.minimum(x, (1 << 32) - x).clamp(min=1).double() * 2.0 ** -32
        q = torch.special.ndtri(u)
        return torch.where(x >= 1 << 31, -q, q)

    lf = N = e = pp = ii = None
    live = None
    tau = float(m.taus[0])
    val = torch.zeros(n, K * I, dtype=torch.float64, device=DEV)
    for s in range(1, n):
        lf1, N1 = starts[s - 1]
        new = (lf1[:, p], N1[p], torch.full_like(p, s - 1), p, i)
        if lf is None:
            lf, N, e, pp, ii = new
        else:
            lf, N, e, pp, ii = (torch.cat((a, b), -1)
                                for a, b in zip((lf, N, e, pp, ii), new))
        zs = normals(s, e, pp, ii)
        _, _, f, D, lfn = next(iter(_evolve64(m, lf, lambda _: zs, A, s, N)))
        v0, v1, v2, x, _ = _date64(m, s, f, D)
        stop = x > _estimate64(m, s, torch.stack((v0, v1, v2)), x, rule)
        val[e[stop], (pp * I + ii)[stop]] = (x / N)[stop]
        live = ~stop
        lf, N = lfn[1:][:, live], (N * (1.0 + tau * f[0]))[live]
        e, pp, ii = e[live], pp[live], ii[live]
    Q = val.view(n, K, I).mean(2)
    Q[n - 1] = 0.0
    # duality gap: the exercise values are the rebates
    best, bal, low = (torch.zeros(K, dtype=torch.float64, device=DEV) for _ in range(3))
    done = torch.zeros(K, dtype=torch.bool, device=DEV)
    for s in range(n):
        hit = X[s] > 0
        best = torch.maximum(best, torch.where(hit, -bal, Z[s] - Q[s] - bal))
        bal = torch.where(hit, bal + Z[s] - Q[s], bal)
        low = torch.where(hit & ~done, Z[s], low)
        done = done | hit
    best = torch.maximum(best, -bal)

    def mean_se(x):
        return x.mean(), ((x * x).mean() - x.mean() ** 2).clamp(min=0.0).sqrt() / math.sqrt(K)

    (gap, gap_se), (lower, lower_se) = mean_se(best), mean_se(low)
    return {"lower": lower, "lower_se": lower_se, "gap": gap, "gap_se": gap_se, "Q": Q, "Z": Z,
            "X": None}


def exact(case, seed):
    kind, m = case["kind"], _market(case, seed)
    if kind == "strip":
        return _payoffs64(m, case["paths"], case["offset"], None)[0]
    if kind in ("price", "staged"):
        return _price64(case, m, None)
    if kind == "nested":
        return _price64(case, m, Selector.production(case["depth"]))
    if kind == "inputs":
        vars_, ex, cf, num = _first_pass64(m, case["paths"], case["offset"])
        return {"vars": vars_, "ex": ex, "cf": cf, "num": num}
    if kind == "regress":
        ls = _ls_inputs(m, case["paths"], 0)
        r = _regress64(m, ls.vars, ls.ex, ls.cf, ls.num)
        return {"beta": r["beta"][:, 0], "means": r["means"][:, 0], "sds": r["sds"][:, 0],
                "price": r["price"].reshape(1), "status": None}
    rule = _rule64(_frozen_rule(m)) if len(m.ex_steps) else None
    if kind == "greeks":
        return _greeks64(case, m, rule)
    return _bound64(case, m, rule, 20240601 + seed)
