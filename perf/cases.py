"""Performance cases of the pricing engine: the calls a user's program makes.

    listed()             the standing cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what the program holds before the call
    run(state)           one pass through the public entry points
    work(case)           the bytes and operations of one pass
    exact(case, seed)    the same outputs in 64-bit torch / numpy

A case names a kind and its sizes and options; the market parameters and the
Philox seed come from `seed`. The sizes are those of the reference's run
scripts (path counts 10^4 .. 10^8, 200 dates, 4 assets), of bench.py's
workloads and of parcompfin_gb300/workloads.py.

  eur          mc_eur: one European contract, 10^4 .. 2^28 paths
  asia         mc_asia: one Asian contract, 10^4 .. 2^22 paths
  basket       mc_eur_multi / mc_basket: one basket of 2 .. 64 assets
  amer         mc_amer: one American contract by Longstaff-Schwartz
  asia_book    a plan of Asian contracts of uneven N and M, repriced
  basket_book  a plan of baskets with full correlation matrices, repriced
  amer_book    a plan of American puts of equal size, repriced
  mixed_book   a plan of all four kinds, in the served stream's proportions
  binom        binom_embar_batch: closed binomial sums of uneven N
  lattice      binom_vanilla_eur / _amer: backward induction on one lattice
"""
import math
import random

import numpy as np
import torch

import parcompfin_gb300 as pcf

RESULT = np.dtype([("price", "f8"), ("std_error", "f8"), ("price_plain", "f8"),
                   ("std_error_plain", "f8"), ("price_cv", "f8"), ("std_error_cv", "f8"),
                   ("cv_beta", "f8"), ("cv_mean", "f8"), ("discount", "f8"), ("sums", "f8", 5),
                   ("n_paths", "i8")])


def listed():
    return [
        # A quote on one European call at the path count of a quick look: what
        # it costs is the call itself (launches, copies, the wait).
        dict(name="eur_100k", kind="eur", N=100_000, payoff=1, cv=False),
        # The same contract priced to a cent of a cent: a long run of paths.
        dict(name="eur_2p28", kind="eur", N=1 << 28, payoff=1, cv=False),
        # runscript_mc_asia.sh: one Asian call, 200 monitoring dates.
        dict(name="asia_1m_m200", kind="asia", N=1_000_000, M=200, payoff=1, mode=0, cv=False),
        # runscript_mc_eur_multi.sh: one basket of four equicorrelated assets.
        dict(name="basket_1m_d4", kind="basket", N=1_000_000, d=4, payoff=1, full=False, cv=False),
        # runscript_mc_amer.sh's middle: one American option, 200 dates.
        dict(name="amer_100k_m200", kind="amer", N=100_000, M=200, payoff=-1, ref=False, cv=True),
        # bench.py --workload lsm: one large American put.
        dict(name="amer_1m_m50", kind="amer", N=1 << 20, M=50, payoff=-1, ref=False, cv=True),
        # bench.py --workload asia: a book of 256 Asian calls, M in {12, 52,
        # 252}, N uneven, with the geometric control variate.
        dict(name="asia_book_256", kind="asia_book", n=256, Nlo=1 << 16, Nhi=1 << 22),
        # bench.py --workload basket: index baskets of 4, 16 and 64 assets.
        dict(name="basket_book", kind="basket_book", d0=4, d1=16, d2=64, N=1 << 22, cv=False),
        # bench.py --workload amerbatch: 64 American puts with their control
        # variate, as a market maker reprices a strike ladder.
        dict(name="amer_book_64", kind="amer_book", n=64, N=1 << 16, M=50),
        # bench.py's default stream: 1000 requests of all kinds at the path
        # counts that 5e-4 relative standard error asks for.
        dict(name="mixed_book_1000", kind="mixed_book", n=1000),
        # bench.py --workload binom: 1024 closed binomial sums, N in 1e3..2e5.
        dict(name="binom_1024", kind="binom", n=1024, Nlo=1_000, Nhi=200_000, mode="reference"),
        # The lattice price that runscript_mc_amer.sh compares against.
        dict(name="lattice_amer_10k", kind="lattice", N=10_000, payoff=-1, american=True),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["eur", "asia", "basket", "amer", "asia_book", "basket_book", "amer_book",
                       "mixed_book", "binom", "lattice"])
    pf = rng.choice([1, -1])
    if kind == "eur":
        return dict(kind=kind, N=_log_int(rng, 10_000, 1 << 28), payoff=pf, cv=rng.random() < 0.5)
    if kind == "asia":
        return dict(kind=kind, N=_log_int(rng, 10_000, 1 << 22), M=rng.choice([12, 52, 200, 252, rng.randint(5, 260)]),
                    payoff=pf, mode=rng.choice([0, 0, 1]), cv=rng.random() < 0.5)
    if kind == "basket":
        return dict(kind=kind, N=_log_int(rng, 10_000, 1 << 22), d=_log_int(rng, 2, 64), payoff=pf,
                    full=rng.random() < 0.5, cv=rng.random() < 0.5)
    if kind == "amer":
        M = rng.choice([12, 50, 200, rng.randint(10, 200)])
        hi = min(1 << 21, (1 << 20) * 100 // M)
        return dict(kind=kind, N=2 * (_log_int(rng, 10_000, hi) // 2), M=M, payoff=pf,
                    ref=rng.random() < 0.3, cv=rng.random() < 0.5)
    if kind == "asia_book":
        return dict(kind=kind, n=_log_int(rng, 16, 256), Nlo=1 << 16, Nhi=_log_int(rng, 1 << 18, 1 << 22))
    if kind == "basket_book":
        d = sorted(rng.sample(range(2, 65), 3))
        return dict(kind=kind, d0=d[0], d1=d[1], d2=d[2], N=_log_int(rng, 1 << 16, 1 << 22),
                    cv=rng.random() < 0.5)
    if kind == "amer_book":
        return dict(kind=kind, n=_log_int(rng, 4, 64), N=2 * (_log_int(rng, 1 << 14, 1 << 17) // 2),
                    M=rng.choice([25, 50, rng.randint(12, 60)]))
    if kind == "mixed_book":
        return dict(kind=kind, n=_log_int(rng, 50, 1000))
    if kind == "binom":
        lo = _log_int(rng, 1_000, 20_000)
        return dict(kind=kind, n=_log_int(rng, 1, 1024), Nlo=lo, Nhi=max(lo, _log_int(rng, 2_000, 200_000)),
                    mode=rng.choice(["reference", "reference", "accurate"]))
    return dict(kind=kind, N=_log_int(rng, 100, 20_000), payoff=pf, american=rng.random() < 0.5)


# ---- the contracts of a case -------------------------------------------------


def _wishart_corr(d, seed):
    """0.7 (all pairs 0.3) + 0.3 (normalised Wishart with d + 2 degrees)."""
    x = np.random.default_rng(seed).standard_normal((d, d + 2))
    w = x @ x.T
    s = np.sqrt(np.diag(w))
    c = 0.7 * 0.3 + 0.3 * (w / np.outer(s, s))
    c = 0.5 * (c + c.T)
    np.fill_diagonal(c, 1.0)
    return c.tolist()


def _amer_put(rng, N, M, i):
    return dict(method="amer", S0=100.0, E=rng.uniform(90, 110), r=0.05, sigma=rng.uniform(0.2, 0.4),
                T=1.0, N=N, payoff_fun=-1, M=M, use_cv=True, stream=i)


def _asia_call(rng, N, i):
    return dict(method="asia", S0=100.0, E=rng.uniform(90, 110), r=0.04, sigma=rng.uniform(0.15, 0.4),
                T=rng.uniform(0.5, 2.0), N=N, payoff_fun=1, M=rng.choice([12, 52, 252]), use_cv=True,
                stream=i)


def _contracts(case, seed):
    """The case's contracts: keyword arguments of pcf.request() for the Monte
    Carlo kinds, argument tuples for the binomial ones."""
    rng = random.Random("%s %d" % (case["kind"], seed))
    kind = case["kind"]
    if kind == "eur":
        out = [dict(method="eur", S0=100.0, E=100.0 * rng.uniform(0.9, 1.1), r=rng.uniform(0.02, 0.06),
                    sigma=rng.uniform(0.15, 0.75), T=rng.uniform(0.5, 1.5), N=case["N"],
                    payoff_fun=case["payoff"], use_cv=case["cv"])]
    elif kind == "asia":
        out = [dict(method="asia", S0=100.0, E=rng.uniform(90, 110), r=rng.uniform(0.02, 0.05),
                    sigma=rng.uniform(0.15, 0.75), T=rng.uniform(0.5, 2.0), N=case["N"], M=case["M"],
                    payoff_fun=case["payoff"], mode=case["mode"], use_cv=case["cv"])]
    elif kind == "basket":
        d = case["d"]
        q = dict(method="basket", S0=100.0, E=rng.uniform(95, 105), r=rng.uniform(0.02, 0.1),
                 sigma=rng.uniform(0.15, 0.35), T=1.0, N=case["N"], payoff_fun=case["payoff"], assets=d,
                 rho=rng.uniform(0.2, 0.6), use_cv=case["cv"], scale_by_sqrt_T=False)
        if case["full"]:
            q.update(basket_S0=[100.0 * rng.uniform(0.9, 1.1) for _ in range(d)],
                     basket_sigma=[rng.uniform(0.15, 0.35) for _ in range(d)],
                     corr=_wishart_corr(d, seed), scale_by_sqrt_T=True)
        out = [q]
    elif kind == "amer":
        out = [dict(method="amer", S0=100.0, E=rng.uniform(90, 110), r=rng.uniform(0.02, 0.06),
                    sigma=rng.uniform(0.2, 0.75), T=1.0, N=case["N"], M=case["M"],
                    payoff_fun=case["payoff"], mode=int(case["ref"]), use_cv=case["cv"])]
    elif kind == "asia_book":
        lo, hi = math.log2(case["Nlo"]), math.log2(case["Nhi"])
        # The N of a book, one in each of n strata of the logarithm, so that
        # books of the same case hold the same work.
        Ns = [int(2 ** (lo + (hi - lo) * (k + 0.5) / case["n"])) for k in range(case["n"])]
        rng.shuffle(Ns)
        out = [_asia_call(rng, N, i) for i, N in enumerate(Ns)]
        for i, q in enumerate(sorted(out, key=lambda q: q["N"])):
            q["M"] = (12, 52, 252)[i % 3]
    elif kind == "basket_book":
        out = [dict(method="basket", S0=100.0, E=100.0, r=0.03, sigma=0.25, T=1.0, N=case["N"],
                    payoff_fun=1, assets=d, basket_S0=[100.0] * d,
                    basket_sigma=[rng.uniform(0.15, 0.35) for _ in range(d)],
                    corr=_wishart_corr(d, seed + d), use_cv=case["cv"], stream=i)
               for i, d in enumerate((case["d0"], case["d1"], case["d2"]))]
    elif kind == "amer_book":
        out = [_amer_put(rng, case["N"], case["M"], i) for i in range(case["n"])]
    elif kind == "mixed_book":
        out = []
        for i in range(case["n"]):
            u = i % 10  # 30 % European, 20 % basket, 30 % Asian, 20 % American
            if u < 3:
                out.append(dict(method="eur", S0=100.0, E=100.0 * rng.uniform(0.9, 1.1),
                                r=0.05 * rng.uniform(0.8, 1.2), sigma=0.2 * rng.uniform(0.8, 1.2),
                                T=rng.uniform(0.8, 1.2), N=int(2 ** rng.uniform(18, 22)), payoff_fun=1,
                                use_cv=True, stream=i))
            elif u < 5:
                d = rng.randint(2, 32)
                out.append(dict(method="basket", S0=100.0, E=100.0, r=0.03, sigma=0.25, T=1.0,
                                N=int(2 ** rng.uniform(14, 18)), payoff_fun=1, assets=d, rho=0.3,
                                basket_sigma=[rng.uniform(0.15, 0.35) for _ in range(d)], use_cv=True,
                                stream=i))
            elif u < 8:
                out.append(_asia_call(rng, int(2 ** rng.uniform(13, 17)), i))
            else:
                out.append(_amer_put(rng, 1 << 16, 50, i))
    elif kind == "binom":
        return [(100.0, rng.uniform(80, 120), rng.uniform(0.01, 0.06), rng.uniform(0.1, 0.5),
                 rng.uniform(0.25, 2.0), rng.randint(case["Nlo"], case["Nhi"]), rng.choice([1, -1]))
                for _ in range(case["n"])]
    else:
        return [(100.0, rng.uniform(90, 110), rng.uniform(0.02, 0.06), rng.uniform(0.2, 0.75),
                 rng.uniform(0.5, 1.5), case["N"], case["payoff"])]
    for q in out:
        q["seed"] = seed
    return out


# ---- the calls ---------------------------------------------------------------


class _Book:
    """A plan that goes with its last reference."""

    def __init__(self, reqs):
        self.plan = pcf.Plan(reqs)

    def __del__(self):
        self.plan.close()


def prepare(case, seed):
    qs = _contracts(case, seed)
    if case["kind"].endswith("_book"):
        return dict(kind="book", book=_Book([pcf.request(**q) for q in qs]))
    if case["kind"] == "binom":
        return dict(kind="binom", contracts=qs, mode=case["mode"])
    if case["kind"] == "lattice":
        fn = pcf.binom_vanilla_amer if case["american"] else pcf.binom_vanilla_eur
        return dict(kind="lattice", fn=fn, args=qs[0])
    q = qs[0]
    args = (q["S0"], q["E"], q["r"], q["sigma"], q["T"], q["N"])
    more = dict(seed=q["seed"], use_cv=q["use_cv"])
    if case["kind"] == "eur":
        fn, args = pcf.mc_eur_result, args + (q["payoff_fun"],)
    elif case["kind"] == "asia":
        fn, args = pcf.mc_asia_result, args + (q["M"], q["payoff_fun"])
        more["mode"] = q["mode"]
    elif case["kind"] == "amer":
        fn, args = pcf.mc_amer_result, args + (q["M"], q["payoff_fun"])
        more["ref_exercise"] = bool(q["mode"])
    elif case["full"]:
        fn = pcf.mc_basket_result
        args = (q["basket_S0"], q["basket_sigma"], q["corr"], q["r"], q["T"], q["E"], q["N"],
                q["payoff_fun"])
    else:
        fn, args = pcf.mc_eur_multi_result, args + (q["payoff_fun"], q["assets"], q["rho"])
    return dict(kind="single", fn=fn, args=args, more=more)


def _fields(results):
    a = np.frombuffer(b"".join(map(bytes, results)), RESULT)
    return {k: a[k] for k in RESULT.names}


def run(state):
    if state["kind"] == "book":
        state["book"].plan.launch()
        return _fields(state["book"].plan.results())
    if state["kind"] == "single":
        return _fields([state["fn"](*state["args"], **state["more"])])
    if state["kind"] == "binom":
        return np.array(pcf.binom_embar_batch(state["contracts"], mode=state["mode"]))
    return np.array([state["fn"](*state["args"])])


# ---- what a pass cannot do without -------------------------------------------


def work(case):
    """Bytes: each contract's parameters in, its results out. Operations: per
    path, step or date the generator's multiplies and logic (15 a normal), the
    transform to normals (8 a normal) and the model's own arithmetic; per
    binomial term two exponentials and two powers of a 53-bit number (20
    operations each); per lattice node two products, a sum and a quotient
    (with the exercise value's product, difference and two maxima)."""
    if case["kind"] == "lattice":
        N = case["N"]
        return {"bytes": 56 + 8, "flops": (N + 1) * (N + 2) / 2 * (8.0 if case["american"] else 4.0)}
    qs = _contracts(case, 1)
    if case["kind"] == "binom":
        return {"bytes": len(qs) * (48 + 8), "flops": sum(min(q[5], 16 * math.sqrt(q[5])) * 85 for q in qs)}
    b = f = 0.0
    for q in qs:
        b += 60 + RESULT.itemsize
        if q["method"] == "eur":
            f += q["N"] * (23.0 + (10 if q["use_cv"] else 7))
        elif q["method"] == "asia":
            f += q["N"] * (q["M"] * (23.0 + (8 if q["use_cv"] else 6)) + 10)
        elif q["method"] == "basket":
            d = q["assets"]
            b += 8.0 * d * (d + 2)
            f += q["N"] * (d * 23.0 + d * (d + 1) + 4 * d + 10)
        else:  # a normal drives two paths; a path-date: step, regression sums, decision
            f += q["N"] * (q["M"] * (11.5 + 5 + 14 + 6) + 20.0)
    return {"bytes": b, "flops": f}


# ---- the same outputs in 64 bits ---------------------------------------------

DEV = "cuda" if torch.cuda.is_available() else "cpu"
CHUNK = 1 << 23  # values a chunk of paths holds at once


def _normals(seed, stream, tag, x, y):
    """Four standard normals for each x (int64 tensor): Philox4x32-10 words
    of counter (x lo, y, stream, tag << 16 | x hi), then Box-Muller."""
    m = 0xFFFFFFFF
    c = [x & m, torch.full_like(x, y), torch.full_like(x, stream), (x >> 32) | (tag << 16)]
    k0, k1 = seed & m, (seed >> 32) & m
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57  # mod 2^64
        c = [((p1 >> 32) & m) ^ c[1] ^ k0, p1 & m, ((p0 >> 32) & m) ^ c[3] ^ k1, p0 & m]
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    u = [((w >> 9) * 2 + 1).double() * 2.0 ** -24 for w in c]
    z = []
    for a, t in ((u[0], u[1]), (u[2], u[3])):
        r = torch.sqrt(-2.0 * torch.log(a))
        th = math.pi * (2.0 * t - 1.0)
        z += [r * torch.cos(th), r * torch.sin(th)]
    return z


def _cdf(x):
    return 0.5 * math.erfc(-x / math.sqrt(2.0))


def _lognormal_mean(mu, var, K, pf):
    """E max(pf (X - K), 0) of X = e^{N(mu, var)}."""
    fwd = math.exp(mu + 0.5 * var)
    if var <= 0 or K <= 0:
        return max(pf * (fwd - K), 0.0)
    sd = math.sqrt(var)
    d1 = (mu - math.log(K) + var) / sd
    return pf * (fwd * _cdf(pf * d1) - K * _cdf(pf * (d1 - sd)))


def _estimate(s, n, mu, disc, cv, n_paths, floor=0.0):
    s = [float(v) for v in s]
    nan = float("nan")
    y = s[0] / n
    vy = max((s[1] - n * y * y) / (n - 1), 0.0)
    out = dict(price_plain=max(disc * y, floor), std_error_plain=disc * math.sqrt(vy / n), price_cv=nan,
               std_error_cv=nan, cv_beta=0.0, cv_mean=mu, discount=disc, sums=s, n_paths=n_paths)
    if cv:
        g = s[2] / n
        vg, cov = (s[3] - n * g * g) / (n - 1), (s[4] - n * y * g) / (n - 1)
        out["cv_beta"] = cov / vg
        out["price_cv"] = max(disc * (y - cov / vg * (g - mu)), floor)
        out["std_error_cv"] = disc * math.sqrt(max(vy - cov * cov / vg, 0.0) / n)
    out["price"], out["std_error"] = ((out["price_cv"], out["std_error_cv"]) if cv else
                                      (out["price_plain"], out["std_error_plain"]))
    return out


def _moments(y, g, cv):
    z = torch.zeros((), dtype=torch.float64, device=DEV)
    return torch.stack([y.sum(), (y * y).sum()] + ([g.sum(), (g * g).sum(), (y * g).sum()] if cv else [z, z, z]))


def _exact_paths(q):
    """European, Asian and basket contracts: chunks of paths."""
    S0, E, r, sig, T, N, pf = (q[k] for k in ("S0", "E", "r", "sigma", "T", "N", "payoff_fun"))
    seed, stream, cv = q["seed"], q.get("stream", 0), q["use_cv"]
    tot = torch.zeros(5, dtype=torch.float64, device=DEV)
    pay = lambda s: torch.clamp(pf * (s - E), min=0.0)  # noqa: E731
    if q["method"] == "eur":
        mu = S0 * math.exp(r * T)
        nu, vol = (r - 0.5 * sig * sig) * T, sig * math.sqrt(T)
        step = CHUNK // 4
        for q0 in range(0, (N + 3) // 4, step):
            x = torch.arange(q0, min(q0 + step, (N + 3) // 4), device=DEV)
            z = torch.stack(_normals(seed, stream, 1, x, 0), 1).reshape(-1)[: N - 4 * q0]
            s = S0 * torch.exp(nu + vol * z)
            tot += _moments(pay(s), s, cv)
    elif q["method"] == "asia":
        M, mode = q["M"], q.get("mode", 0)
        dt = T / M
        w = [1.0 / M] * (M + 1)
        w[0] = 0.5 / M if mode == 0 else 0.0
        w[M] = 0.5 / M if mode == 0 else 1.0 / M
        nu, tail, var, mean = r - 0.5 * sig * sig, 0.0, 0.0, math.log(S0)
        for m in range(M, 0, -1):
            tail += w[m]
            var += dt * tail * tail
            mean += nu * w[m] * m * dt
        mu = _lognormal_mean(mean, var * sig * sig, E, pf)
        for n0 in range(0, N, CHUNK):
            x = torch.arange(n0, min(n0 + CHUNK, N), device=DEV)
            L = torch.zeros(x.numel(), dtype=torch.float64, device=DEV)
            acc, geo = torch.zeros_like(L), torch.zeros_like(L)
            for m in range(M):
                if m % 4 == 0:
                    z = _normals(seed, stream, 2, x, m // 4)
                zm = z[m % 4]
                if mode == 0:
                    acc += torch.exp(L) * (1 + r * dt / 2 + sig * math.sqrt(dt) / 2 * zm)
                L += nu * dt + sig * math.sqrt(dt) * zm
                if mode == 1:
                    acc += torch.exp(L)
                geo += w[m + 1] * L
            tot += _moments(pay(acc * (S0 / M)), pay(S0 * torch.exp(geo)), cv)
    else:
        d = q["assets"]
        s0 = np.array(q.get("basket_S0") or [S0] * d)
        sg = np.array(q.get("basket_sigma") or [sig] * d)
        C = np.array(q["corr"]) if q.get("corr") else np.full((d, d), q["rho"])
        np.fill_diagonal(C, 1.0)
        ts = math.sqrt(T) if q.get("scale_by_sqrt_T", True) else 1.0
        mean = float(np.mean(np.log(s0) + (r - 0.5 * sg * sg) * T))
        mu = _lognormal_mean(mean, float(sg @ C @ sg) / d ** 2 * ts * ts, E, pf)
        Lt = torch.tensor(np.linalg.cholesky(C).T.copy(), device=DEV)
        l0 = torch.tensor(np.log(s0) + (r - 0.5 * sg * sg) * T, device=DEV)
        v = torch.tensor(sg * ts, device=DEV)
        step = CHUNK // d
        for n0 in range(0, N, step):
            x = torch.arange(n0, min(n0 + step, N), device=DEV)
            z = torch.stack([t for a in range((d + 3) // 4) for t in _normals(seed, stream, 3, x, a)][:d], 1)
            ls = l0 + v * (z @ Lt)
            tot += _moments(pay(torch.exp(ls).mean(1)), pay(torch.exp(ls.mean(1))), cv)
    return _estimate(tot.tolist(), N, mu, math.exp(-r * T), cv, N)


def _exact_amer(q):
    """Longstaff-Schwartz on N/2 antithetic pairs, basis {1, u, u^2} of
    u = pf (S - E) / E, over the paths in the money."""
    S0, E, r, sig, T, N, M, pf = (q[k] for k in ("S0", "E", "r", "sigma", "T", "N", "M", "payoff_fun"))
    seed, stream, ref, cv = q["seed"], q.get("stream", 0), q.get("mode", 0), q["use_cv"]
    H, dt = N // 2, T / M
    x = torch.arange(H, device=DEV)
    L = torch.full((2, H), math.log(S0 / E), dtype=torch.float64, device=DEV)
    u = torch.empty((M, 2, H), dtype=torch.float64, device=DEV)
    sgn = torch.tensor([[1.0], [-1.0]], dtype=torch.float64, device=DEV)
    for m in range(M):
        if m % 4 == 0:
            z = _normals(seed, stream, 4, x, m // 4)
        L += (r - 0.5 * sig * sig) * dt + sig * math.sqrt(dt) * sgn * z[m % 4]
        u[m] = torch.clamp(pf * (torch.exp(L) - 1.0), min=0.0)
    disc = [math.exp(-r * dt * k) for k in range(M + 1)]
    cash = u[M - 1] * (E * disc[M])  # discounted to 0
    tau = torch.full((2, H), M, dtype=torch.int64, device=DEV)
    for m in range(M - 1, 0, -1):
        um = u[m - 1]
        itm = um > 0
        i = itm.double()
        y = cash / disc[m] * i
        u2 = um * um
        a = [i.sum(), um.sum(), u2.sum(), (u2 * um).sum(), (u2 * u2).sum(), y.sum(), (y * um).sum(),
             (y * u2).sum()]
        # {1, u, u^2} scaled by the root mean square of u
        k = torch.sqrt(a[2] / torch.clamp(a[0], min=1.0))
        k = torch.where(k > 0, k, torch.ones_like(k))
        b = [a[j] / k ** j for j in range(5)] + [a[5 + j] / k ** j for j in range(3)]
        c00, c01, c02 = b[2] * b[4] - b[3] ** 2, b[2] * b[3] - b[1] * b[4], b[1] * b[3] - b[2] ** 2
        c11, c12, c22 = b[0] * b[4] - b[2] ** 2, b[1] * b[2] - b[0] * b[3], b[0] * b[2] - b[1] ** 2
        det = b[0] * c00 + b[1] * c01 + b[2] * c02
        w = um / k
        fit = ((c00 * b[5] + c01 * b[6] + c02 * b[7]) + (c01 * b[5] + c11 * b[6] + c12 * b[7]) * w +
               (c02 * b[5] + c12 * b[6] + c22 * b[7]) * w * w) / det
        few = a[0] <= 2
        cont = torch.where(few, cash / disc[m], fit)
        ex = torch.where(few | (ref == 0), um * E, torch.clamp(E * um - pf * E, min=0.0))
        go = itm & (ex > cont)
        cash = torch.where(go, ex * disc[m], cash)
        tau = torch.where(go, torch.full_like(tau, m), tau)
    if ref:
        g = u[M - 1] * (E * disc[M])
    else:
        df = torch.tensor(disc, dtype=torch.float64, device=DEV)[tau]
        S = E + pf * cash / df
        rem = (M - tau).double() * dt
        sd = sig * torch.sqrt(torch.clamp(rem, min=1e-300))
        dK = E * torch.exp(-r * rem)
        d1 = (torch.log(S / E) + (r + 0.5 * sig * sig) * rem) / sd
        cdf = lambda t: 0.5 * torch.special.erfc(-t / math.sqrt(2.0))  # noqa: E731
        g = torch.where(tau == M, cash, df * pf * (S * cdf(pf * d1) - dK * cdf(pf * (d1 - sd))))
    s = _moments(cash.mean(0), g.mean(0), True).tolist()
    mu = math.exp(-r * T) * _lognormal_mean(math.log(S0) + (r - 0.5 * sig * sig) * T, sig * sig * T, E, pf)
    return _estimate(s, H, mu, 1.0, cv, N, max(pf * (S0 - E), 0.0))


def _lattice_constants(r, sig, T, N):
    dt = T / N
    beta = 0.5 * (math.exp(-r * dt) + math.exp((r + sig * sig) * dt))
    u, d = beta + math.sqrt(beta * beta - 1), beta - math.sqrt(beta * beta - 1)
    R = math.exp(r * dt)
    p = (R - d) / (u - d)
    return u, d, p, 1 - p, R


def _exact_binom(contracts, mode):
    """Every pair index i of the binomial sum within 9 sqrt(N) of the weights'
    centres. "reference": log C(N, i) by one FP64 accumulator, + log n for
    n = N .. i+1, then - log j for j = 2 .. N-i, as the method defines it."""
    top = max(q[5] for q in contracts)
    logs = np.array([-math.inf] + [math.log(n) for n in range(1, top + 1)])
    if mode == "accurate":
        lfac = np.concatenate([[0.0], np.cumsum(np.log(np.arange(1, top + 1, dtype=np.longdouble)))])
    idx, acc, end = [], [], []
    for S0, E, r, sig, T, N, pf in contracts:
        u, d, p, _, R = _lattice_constants(r, sig, T, N)
        ps, w = p * u / R, 9 * math.sqrt(N) + 10
        lo = max(0, int(min(N * min(p, ps), N * (1 - max(p, ps))) - w))
        i = np.arange(lo, N // 2 + (1 if N % 2 == 0 else 0) + N % 2)
        if mode == "accurate":
            a = (lfac[N] - lfac[i] - lfac[N - i])
        else:
            down = np.add.accumulate(logs[N:0:-1])  # down[k]: log N + .. + log(N - k)
            a = np.where((i == 0) | (i == N), 0.0, down[np.clip(N - 1 - i, 0, N - 1)])
        idx.append(i)
        acc.append(a)
        end.append(np.where((i == 0) | (i == N), 0, N - i))
    if mode == "reference":
        a, e = np.concatenate(acc), np.concatenate(end)
        order = np.argsort(-e, kind="stable")
        t = torch.tensor(a[order], device=DEV)
        e = e[order]
        alive = np.searchsorted(-e, -np.arange(int(e[0]) + 1), side="right").tolist()  # terms with end >= j
        lg = logs.tolist()
        for j in range(2, int(e[0]) + 1):
            t[: alive[j]].sub_(lg[j])
        back = np.empty_like(a)
        back[order] = t.cpu().numpy()
        acc = np.split(back, np.cumsum([len(i) for i in idx])[:-1])
    out = []
    for (S0, E, r, sig, T, N, pf), i, a in zip(contracts, idx, acc):
        u, d, p, q, R = _lattice_constants(r, sig, T, N)
        lp, lq = math.log(p), math.log(q)
        j = N - i
        su, sd = S0 * np.power(u, i.astype(float)) * np.power(d, j.astype(float)), S0 * np.power(u, j.astype(float)) * np.power(d, i.astype(float))
        if mode == "accurate":
            lp, lq = np.log(np.longdouble(p)), np.log(np.longdouble(q))
        t1 = np.exp((a + i * lp + j * lq).astype(float)) * np.maximum(pf * (su - E), 0.0)
        t2 = np.exp((a + j * lp + i * lq).astype(float)) * np.maximum(pf * (sd - E), 0.0)
        t2 = np.where(2 * i == N, 0.0, t2)
        out.append(math.exp(-r * T) * math.fsum((t1 + t2).tolist()))
    return np.array(out)


def _exact_lattice(S0, E, r, sig, T, N, pf, american):
    u, d, p, q, R = _lattice_constants(r, sig, T, N)
    up = np.array([S0 * math.pow(u, i) for i in range(N + 1)])
    dn = np.array([math.pow(d, i) for i in range(N + 1)])
    pay = lambda n: np.maximum(pf * (up[: n + 1] * dn[n::-1] - E), 0.0)  # noqa: E731
    v = pay(N)
    for n in range(N - 1, -1, -1):
        v = (p * v[1:] + q * v[:-1]) / R
        if american:
            v = np.maximum(v, pay(n))
    return np.array([v[0]])


def exact(case, seed):
    qs = _contracts(case, seed)
    if case["kind"] == "binom":
        return _exact_binom(qs, case["mode"])
    if case["kind"] == "lattice":
        return _exact_lattice(*qs[0], case["american"])
    if sum(q["N"] * q["M"] for q in qs if q["method"] == "asia") > 3e9:
        return None  # over 20 seconds
    got = [_exact_amer(q) if q["method"] == "amer" else _exact_paths(q) for q in qs]
    return {k: np.array([g[k] for g in got], dtype=np.int64 if k == "n_paths" else np.float64)
            for k in RESULT.names}
