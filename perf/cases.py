"""The work a user of keldy_b200 has it do, as timed cases: perturbation series by quasi-Monte
Carlo in one call or one plan, replicas for an error bar, integrand values at given times, the
binned observables, the kernel method, and the training of a learned warper. Sizes are those of
the repository's own benchmark and tests (point counts of the largest workloads cut down).
"""
import math

import numpy as np
import torch

from keldy_b200 import capi, rqmc

# Where a case's table of g^<, g^> comes from: "host", the band integral of a dot between flat
# leads of half-bandwidth 10, summed here and uploaded; "gpu", the framework's flat-band builder.
_CHARGE = dict(path="charge", table="gpu", lo=1, hi=1, points=1000, models=1, replicas=0, flow="", warper="plasma",
               t=20.0, mesh=40001, beta=50.0, bias=0.0, eps=0.0, cubic=False, plan=True, bins=0)


def _charge(name, **kw):
    return dict(_CHARGE, name=name, **kw)


def listed():
    return [
        # one small call of a low order, where the latency of the call counts: an interactive look
        # at the integral, the first rung of a convergence ladder
        _charge("call_order2_1000", table="host", lo=2, hi=2, points=1000, warper="uniform", t=10.0, mesh=10001, plan=False),
        # the plain method at its small size: orders 1..4 of the charge at t = 10, in one call
        _charge("orders1to4_2e16", table="host", lo=1, hi=4, points=1 << 16, warper="uniform", t=10.0, mesh=10001, plan=False),
        # an estimate with an error bar: 16 digital shifts of an odd number of points each
        _charge("replicas_order6", lo=6, hi=6, points=4001, replicas=16, plan=False),
        # the same with the learned spline warper at the size where it meets 1e-3 at order 8
        _charge("replicas_order8_spline", lo=8, hi=8, points=1024, replicas=16, flow="spline", plan=False),
        # values of the integrand at times the caller has (its own sampler, a plot, a test)
        dict(path="points", name="points_order5", order=5, points=10007, t=10.0, mesh=10001, beta=50.0),
        # the throughput workload: order 8, 2^20 points, a plan replayed
        _charge("order8_2e20", lo=8, hi=8, points=1 << 20),
        # the batched series: orders 1..10 with uneven costs in one launch
        _charge("orders1to10_2e20", lo=1, hi=10, points=1 << 20),
        # the biased dot at long times, orders 6..12, cubic table interpolation
        _charge("biased_orders6to12_2e18", lo=6, hi=12, points=1 << 18, t=50.0, mesh=100001, beta=100.0, bias=1.0, eps=0.5,
                cubic=True),
        # a parameter sweep: 256 models with a table each, orders 2..10 by model, in one launch
        _charge("sweep_256", lo=2, hi=10, points=1 << 14, models=256, mesh=20001),
        # the charge as a function of time: one integration binned by the earliest vertex time
        _charge("binned_order7", lo=7, hi=7, points=1 << 18, plan=False, bins=100),
        # the Green function of all times at once by the kernel method, orders 2..8
        dict(path="kernel", name="kernel_orders2to8_2e16", table="gpu", lo=2, hi=8, points=1 << 16, t=20.0, mesh=40001,
             beta=50.0, bins=100),
        # training the coupling warper of an order on samples of the plain method
        dict(path="train", name="train_order6", order=6, samples=1 << 16, batch=8192, epochs=4),
    ]


def _log_int(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["call", "series", "series", "plan", "plan", "replicas", "points", "binned", "kernel", "sweep", "train"])
    if kind == "call":
        n = rng.randint(1, 5)
        return dict(_CHARGE, table="host", lo=n, hi=n, points=_log_int(rng, 50, 20000), plan=False, t=10.0, mesh=10001,
                    warper=rng.choice(["uniform", "plasma"]))
    if kind == "series":
        lo, t = rng.randint(1, 4), rng.uniform(5.0, 30.0)
        return dict(_CHARGE, lo=lo, hi=rng.randint(lo, 8), points=_log_int(rng, 1 << 12, 1 << 18), t=t, plan=False,
                    mesh=2 * rng.randint(5000, 20000) + 1, warper=rng.choice(["uniform", "plasma", "plasma"]),
                    cubic=rng.random() < 0.2)
    if kind == "plan":
        n = rng.randint(5, 12)
        return dict(_CHARGE, lo=n, hi=n, points=_log_int(rng, 1 << 10, 1 << (28 - n)), t=rng.uniform(10.0, 50.0),
                    mesh=2 * rng.randint(10000, 50000) + 1, beta=rng.uniform(10.0, 200.0), bias=rng.uniform(0.0, 2.0),
                    eps=rng.uniform(-1.0, 1.0), cubic=rng.random() < 0.3)
    if kind == "replicas":
        n = rng.randint(3, 8)
        return dict(_CHARGE, lo=n, hi=n, points=_log_int(rng, 256, 1 << 15), replicas=rng.choice([8, 16, 16, 32]),
                    flow=rng.choice(["", "spline"]), plan=False)
    if kind == "points":
        return dict(path="points", order=rng.randint(1, 6), points=_log_int(rng, 1, 20000), t=10.0, mesh=10001,
                    beta=rng.uniform(10.0, 100.0))
    if kind == "binned":
        n = rng.randint(2, 8)
        return dict(_CHARGE, lo=n, hi=n, points=_log_int(rng, 1 << 10, 1 << 18), plan=False, bins=rng.randint(10, 400))
    if kind == "kernel":
        lo = rng.randint(1, 6)
        return dict(path="kernel", table="gpu", lo=lo, hi=rng.randint(lo, 9), points=_log_int(rng, 1 << 9, 1 << 16),
                    t=rng.uniform(5.0, 30.0), mesh=2 * rng.randint(5000, 20000) + 1, beta=rng.uniform(10.0, 100.0),
                    bins=rng.randint(10, 200))
    if kind == "sweep":
        lo = rng.randint(2, 5)
        return dict(_CHARGE, lo=lo, hi=rng.randint(lo + 1, 10), points=_log_int(rng, 500, 1 << 14),
                    models=rng.randint(16, 256), mesh=20001)
    return dict(path="train", order=rng.randint(2, 8), samples=_log_int(rng, 1 << 13, 1 << 16), batch=8192,
                epochs=rng.randint(1, 4))


# ------------------------------------------------------------------------- inputs

def _band_table(t_max, mesh, beta, eps):
    """g^<(t) = i int A f e^{-iwt}, g^>(t) = -i int A (1 - f) e^{-iwt} on [-t_max, t_max]: a level at
    eps of width 1, its spectrum A cut at |w| = 10 and normalised (Gauss-Legendre, 600 nodes)."""
    x, w = np.polynomial.legendre.leggauss(600)
    om = 10.0 * x
    a = w / ((om - eps) ** 2 + 1.0)
    a /= a.sum()
    f = 0.5 * (1.0 - np.tanh(0.5 * beta * om))
    t = np.linspace(-t_max, t_max, mesh)[mesh // 2:]
    e = np.exp(-1j * np.outer(t, om))
    less, great = 1j * (e @ (a * f)), -1j * (e @ (a * (1.0 - f)))
    return (np.concatenate([-less[:0:-1].conj(), less]), np.concatenate([-great[:0:-1].conj(), great]))


def _draws(case, seed):
    """What the seed decides: the level's energy, the first Sobol index, the shifts' seeds."""
    r = np.random.default_rng([seed, 2024])
    return {"eps": case.get("eps", 0.0) + 0.05 * r.uniform(-1.0, 1.0), "k_first": 1 + int(r.integers(0, 1 << 20)),
            "shift": 1 + int(r.integers(0, 1 << 20)), "r": r}


def _models(ctx, case, d):
    if case.get("table", "host") == "host":
        return [ctx.model(case["t"], *_band_table(case["t"], case["mesh"], case["beta"], d["eps"]))]
    if case.get("models", 1) == 1:
        params = [(1.0, d["eps"], case.get("bias", 0.0), case["beta"])]
    else:
        params = [(1.0, e + d["eps"], v, b) for b in (10.0, 50.0, 200.0) for v in np.linspace(0.0, 2.0, 8)
                  for e in np.linspace(-1.0, 1.0, 11)][:case["models"]]
    return capi.flatband_models(ctx, params, case["t"], case["mesh"])


def _chain(case):
    t = case["t"]
    if case.get("warper", "plasma") == "uniform":
        return [(capi.WARPER_UNIFORM, t, 0.0)]
    return [(capi.WARPER_PLASMA_UV, t, 0.0), (capi.WARPER_EXPONENTIAL, t, 1.0)]


def prepare(case, seed):
    d = _draws(case, seed)
    ctx = capi.Context(0)
    s = {"case": case, "ctx": ctx, "draws": d}
    if case["path"] == "train":
        n = case["order"]
        s["x"], s["w"] = _samples(case, d["r"])
        s["flow"] = ctx.flow(n, seed=seed & 0xFFFF)
        s["start"] = s["flow"].params()
        return s
    A, B = (case["t"], 0, 0, 0, 0), (case["t"], 0, 1, 0, 0)
    s["models"] = models = _models(ctx, case, d)
    s["ends"] = (A, B)
    if case["path"] == "points":
        s["times"] = _times(case, d["r"])
        return s
    for m in models:
        if case.get("cubic"):
            m.set_interpolation(3)
    s["chain"] = chain = _chain(case)
    orders = range(case["lo"], case["hi"] + 1)
    if case.get("replicas"):
        n = case["lo"]
        s["rngs"] = [ctx.sobol(n, 31, True, False, d["shift"] + i) for i in range(case["replicas"])]
        s["flow"] = None
        if case["flow"]:
            s["flow"] = ctx.flow(n, kind=capi.FLOW_SPLINE)
            s["flow"].set_params((0.3 * d["r"].standard_normal((n, 49))).astype(np.float32))
        return s
    s["rngs"] = rngs = {n: ctx.sobol(n) for n in orders}
    if case.get("models", 1) > 1:
        which = [(models[i], orders[i % len(orders)]) for i in range(len(models))]
    else:
        which = [(models[0], n) for n in orders]
    s["items"] = [dict(model=m, rng=rngs[n], chain=chain, A=A, B=B, order=n, k_first=d["k_first"], n_points=case["points"])
                  for m, n in which]
    if case["path"] == "charge" and case["plan"]:
        s["plan"] = capi.Plan(ctx, s["items"])
    return s


def _times(case, r):
    return r.uniform(0.0, case["t"], (case["points"], case["order"]))


def _samples(case, r):
    """Points of the unit cube with positive weights that fall off from the first corner, as |f J| does."""
    n = case["order"]
    x = r.random((case["samples"], n))
    w = np.exp(-2.0 * x.sum(axis=1)) * (1.0 + 0.5 * np.cos(3.0 * x @ np.arange(1, n + 1)))
    return x, w / w.mean()


def run(state):
    case, ctx = state["case"], state["ctx"]
    if case["path"] == "train":
        state["flow"].set_params(state["start"])
        loss = state["flow"].train(state["x"], state["w"], epochs=case["epochs"], batch=case["batch"], seed=3)
        return {"loss": loss, "params": state["flow"].params()}
    if case["path"] == "points":
        v, dom = state["models"][0].integrand(*state["ends"], state["times"])
        return {"value": v, "in_domain": dom}
    if case["path"] == "kernel":
        res = capi.integrate_kernel(ctx, state["items"], case["bins"], 0.0, case["t"])
        return {"sum": np.array([r[0] for r in res]), "points": np.array([r[1:3] for r in res]),
                "bins": np.array([r[3] for r in res]), "counts": np.array([r[4] for r in res]),
                "dropped": np.array([r[5] for r in res])}
    if case["replicas"]:
        mean, err, means = rqmc.estimate(ctx, state["models"][0], *state["ends"], state["chain"], case["lo"], case["points"],
                                         case["replicas"], k_first=state["draws"]["k_first"], rngs=state["rngs"],
                                         flow=state["flow"])
        return {"means": means, "mean": np.array([mean]), "stderr": err}
    if case["bins"]:
        res = capi.integrate_binned(ctx, state["items"], case["bins"], 0.0, case["t"])
        return {"sum": np.array([r[0] for r in res]), "points": np.array([r[1:4] for r in res]),
                "bins": np.array([r[4] for r in res]), "counts": np.array([r[5] for r in res]),
                "dropped": np.array([r[6] for r in res])}
    res = state["plan"].run() if case["plan"] else capi.integrate(ctx, state["items"])
    return {"sum": np.array([r[0] for r in res]), "points": np.array([r[1:] for r in res])}


# ------------------------------------------------------------- the work of one pass

def _point_flops(n):
    """Complex multiply-adds (8 flops) that the 2^n signed products of determinants of one point
    cannot do without once their eliminations are shared: a node with m vertices left has an
    (m+1)^2 matrix to update for each of its two children."""
    return 8 * sum((1 << (n - m)) * (m + 1) ** 2 for m in range(0, n))


def work(case):
    if case["path"] == "train":
        steps = max(1, case["samples"] // min(case["batch"], case["samples"])) * case["epochs"]
        layers = 18
        # per sample: forward, gradient of the inputs and gradient of the weights of each matrix
        flops = 3 * 2 * layers * 128 * 128 * min(case["batch"], case["samples"]) * steps
        return {"bytes": case["samples"] * (case["order"] + 1) * 8 + 2 * layers * 128 * 128 * 4, "flops": flops}
    if case["path"] == "points":
        n, p = case["order"], case["points"]
        return {"bytes": p * (n * 8 + 16 + 4) + case["mesh"] * 32, "flops": p * _point_flops(n)}
    orders = range(case["lo"], case["hi"] + 1)
    if case.get("models", 1) > 1:
        orders = [orders[i % len(orders)] for i in range(case["models"])]
    mult = max(1, case.get("replicas", 0))
    per = (lambda n: 2 * _point_flops(n)) if case["path"] == "kernel" else _point_flops
    flops = mult * case["points"] * sum(per(n) for n in orders)
    out = len(list(orders)) * mult * (40 + 24 * case.get("bins", 0))
    return {"bytes": case.get("models", 1) * case["mesh"] * 32 + out, "flops": flops}


# -------------------------------------------------------------- the same in plain numpy

_MOST = 4.0e8  # about 20 seconds of small determinants


def exact(case, seed):
    if case["path"] == "train" or case.get("table", "host") != "host" or case.get("replicas"):
        return None
    orders = [case["order"]] if case["path"] == "points" else range(case["lo"], case["hi"] + 1)
    if sum(case["points"] * (1 << n) * (n + 1) ** 2 for n in orders) > _MOST:
        return None
    d = _draws(case, seed)
    table = _band_table(case["t"], case["mesh"], case["beta"], d["eps"])
    if case["path"] == "points":
        t = _times(case, d["r"])
        return {"value": _integrand(case, table, t), "in_domain": None}
    sums = []
    for n in orders:
        eng = torch.quasirandom.SobolEngine(n)
        eng.fast_forward(d["k_first"])
        x = eng.draw(case["points"], dtype=torch.float64).numpy()
        total = 0j
        for part in np.array_split(x, max(1, len(x) >> 14)):
            u, jac = _warp(case, part)
            ok = (u >= 0.0).all(axis=1)
            total += (_integrand(case, table, u[ok]) * jac[ok]).sum()
        sums.append(total)
    return {"sum": np.array(sums), "points": None}


def _warp(case, x):
    t = case["t"]
    if case["warper"] == "uniform":
        return t * x, np.full(len(x), t ** x.shape[1])
    v = t - np.log1p(np.expm1(t) * x)
    jac = np.prod(-np.expm1(-t) * np.exp(v), axis=1)
    return t - np.cumsum(v, axis=1), jac


def _integrand(case, table, u):
    """sum_a (-1)^|a| det(s1_a) det(s2_a) of G^<(t, t) at the times u [points][n], determinant by
    determinant: the contour-ordered g0 between the vertices' chosen copies and the two ends."""
    p, n = u.shape
    t, mesh = case["t"], case["mesh"]
    delta = 2.0 * t / (mesh - 1)

    def both(x):
        a = (x + t) / delta
        i = np.clip(np.floor(a).astype(np.int64), 0, mesh - 2)
        w = a - i
        return [(1.0 - w) * g[i] + w * g[i + 1] for g in table]

    full = np.concatenate([u, np.full((p, 1), t)], axis=1)
    less, great = both(full[:, :, None] - full[:, None, :])
    later = full[:, :, None] > full[:, None, :]
    eq = np.arange(n + 1)
    later[:, n, :], later[:, :, n] = True, False  # the ends lie last on the forward branch, first on the backward one
    fwd = np.where(later, great, less)
    bwd = np.where(later, less, great)
    fwd[:, eq, eq] = bwd[:, eq, eq] = less[:, eq, eq]
    g = np.stack([np.stack([fwd, less], 3), np.stack([great, bwd], 3)], 2)  # [p][i][a][j][b]
    total = np.zeros(p, np.complex128)
    for cfg in range(1 << n):
        a = [(cfg >> i) & 1 for i in range(n)]
        # the row of the end A = (t, forward), the column of the end B = (t, backward)
        m = np.empty((p, n + 1, n + 1), np.complex128)
        for i in range(n):
            for j in range(n):
                m[:, i, j] = g[:, i, a[i], j, a[j]]
            m[:, n, i] = g[:, n, 0, i, a[i]]
            m[:, i, n] = g[:, i, a[i], n, 1]
        m[:, n, n] = 0.0
        term = np.linalg.det(m) * np.linalg.det(m[:, :n, :n])
        total += -term if sum(a) & 1 else term
    return total
