"""The performance cases: what users of dadi_gb300 have it compute, through its public
entry points, from one small 1-D integration to a thousand 2-D spectra.

Kinds of case (`kind`):

* one_pop, split_mig, im, growth3, four_pops: one model evaluation through the drop-in
  (integration.* and models.* with numerics.make_extrap_func), host arrays in and out, as
  dadi's own model code calls it;
* batch: Batch2D.run, many isolation-with-migration (IM) parameter sets at once, with the
  Poisson likelihood (optionally under the delj trick);
* dfe: spectra over a (gamma1, gamma2) grid, as a DFE cache is filled;
* grad: Batch2D.loglik_and_grad, likelihood gradients of IM parameter sets;
* model_batch: ModelBatch.run, three- or four-population parameter sets at once;
* grad_nd: gradients of the three-population growth model by the N-dimensional adjoint.

The IM sets are drawn like the benchmark's (log-uniform sizes and times, uniform migration),
with the ends of the ranges drawn in so that no single set's time loop exceeds 5,000 steps.
"""
import math

import numpy as np
import torch

from dadi_gb300 import adjoint_nd, batch, batchnd, dfe, integration, models, numerics

#: FP64 operations one grid point of one axis sweep cannot do without: the two
#: off-diagonals (2 multiplies, 2 adds), the pivot (multiply, add, divide), the elimination
#: (multiply, add, multiply), the coupling (multiply) and the substitution (multiply, add).
POINT_FLOPS = 13


def listed():
    return [
        # a one-population epoch on one grid: the smallest call there is
        dict(name="one_pop_40", kind="one_pop", pts=40),
        # the two-population tutorial model at the test suite's grids: constant parameters
        dict(name="split_mig_60", kind="split_mig", pts=40, step=10, ns=20),
        # one step of a user's own optimiser over IM at the benchmark's grids
        dict(name="im_100", kind="im", pts=80, step=10, ns=40),
        # the benchmark's workload: spectra and likelihoods of many IM sets, launches shaped
        # per grid as the autotuner shapes them
        dict(name="im_batch_100", kind="batch", n=1000, pts=80, step=10, ns=40,
             mode="per_grid", delj=False),
        # a coarse scan of parameter space on small odd grids, the engine's defaults
        dict(name="im_batch_45", kind="batch", n=257, pts=31, step=7, ns=12,
             mode="persistent", delj=False),
        # fine, ragged grids (large samples), few sets
        dict(name="im_batch_133", kind="batch", n=100, pts=109, step=12, ns=60,
             mode="per_grid", delj=False),
        # the same engine under dadi's delj trick
        dict(name="im_batch_delj_60", kind="batch", n=64, pts=40, step=10, ns=20,
             mode="persistent", delj=True),
        # a DFE cache: selection from nearly neutral to strong
        dict(name="dfe_44", kind="dfe", gammas=7, gmax=60.0, pts=30, step=7, ns=10),
        # likelihood gradients of a population of parameter sets (an ensemble or HMC step)
        dict(name="im_grad_80", kind="grad", n=24, pts=60, step=10, ns=30),
        # one three-population integration on one grid of the three-population workload
        dict(name="growth3_70", kind="growth3", pts=70, ns=20),
        # four populations, several parameter sets together
        dict(name="four_batch_26", kind="model_batch", model="four", n=12, pts=18, step=4, ns=6),
        # gradients of the three-population workload
        dict(name="growth3_grad_40", kind="grad_nd", n=6, pts=40, ns=12),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["one_pop", "split_mig", "im", "batch", "batch", "dfe", "grad", "growth3",
                       "model_batch", "grad_nd"])
    if kind == "one_pop":
        return dict(kind=kind, pts=int(_log(rng, 20, 200)))
    if kind in ("split_mig", "im"):
        pts = int(_log(rng, 24, 100))
        return dict(kind=kind, pts=pts, step=rng.randint(5, 10), ns=rng.randint(8, 40))
    if kind == "batch":
        pts, step = int(_log(rng, 24, 110)), rng.randint(5, 12)
        delj = rng.random() < 0.2
        # no more point-sweeps than the largest listed case; the delj rows cost ten times
        most = 1000 * (90 / (pts + step)) ** 2 / (20 if delj else 1)
        return dict(kind=kind, n=int(_log(rng, 16, max(20, min(1000, most)))), pts=pts,
                    step=step, ns=rng.randint(8, 40),
                    mode=rng.choice(["per_grid", "persistent"]), delj=delj)
    if kind == "dfe":
        return dict(kind=kind, gammas=rng.randint(4, 12), gmax=_log(rng, 10, 120),
                    pts=rng.randint(24, 40), step=rng.randint(5, 9), ns=rng.randint(6, 20))
    if kind == "grad":
        pts = int(_log(rng, 28, 100))
        return dict(kind=kind, n=max(1, int(_log(rng, 1, 24) * min(1.0, (60 / pts) ** 2))),
                    pts=pts, step=rng.randint(5, 10), ns=rng.randint(8, 40))
    if kind == "growth3":
        return dict(kind=kind, pts=int(_log(rng, 20, 90)), ns=rng.randint(6, 20))
    if kind == "model_batch":
        if rng.random() < 0.5:
            return dict(kind=kind, model="four", n=rng.randint(1, 12), pts=rng.randint(10, 18),
                        step=rng.randint(2, 4), ns=rng.randint(3, 6))
        return dict(kind=kind, model="growth3", n=rng.randint(2, 10), pts=rng.randint(24, 44),
                    step=rng.randint(4, 10), ns=rng.randint(6, 16))
    return dict(kind=kind, n=rng.randint(1, 6), pts=rng.randint(16, 44), ns=rng.randint(6, 16))


# ----------------------------------------------------------------- inputs

def _grids(case):
    return [case["pts"] + k * case["step"] for k in range(3)] if "step" in case else [case["pts"]]


def _im_sets(rng, n):
    """IM parameter rows (s, nu1, nu2, T, m12, m21)."""
    s = rng.uniform(0.05, 0.95, n)
    nu = np.exp(rng.uniform(np.log(0.05), np.log(20), (2, n)))
    T = np.exp(rng.uniform(np.log(0.01), np.log(0.5), n))
    m = rng.uniform(0, 10, (2, n))
    return np.stack([s, nu[0], nu[1], T, m[0], m[1]], axis=1)


def _growth3_sets(rng, n):
    base = adjoint_nd.Growth3.from_model_params(models.GROWTH3_DEFAULT)
    th = base * np.exp(rng.uniform(np.log(0.6), np.log(1.6), (n, len(base))))
    th[:, 9] *= 0.25  # an epoch of 0.02-0.06: 100-300 steps
    return th


def _growth3_params(th):
    return (tuple(th[0:3]), tuple(th[3:6]), tuple(th[6:9]), models.GROWTH3_DEFAULT[3], th[9])


def _counts(rng, ns, ndim):
    """An observed spectrum: Poisson counts around theta/(sum of the indices)."""
    i = sum(np.meshgrid(*[np.arange(ns + 1.0)] * ndim, indexing="ij"))
    i.flat[0] = 1
    return rng.poisson(5e3 / i ** ndim).astype(np.float64)


def _inputs(case, seed):
    """The host inputs of a case (what the call's arguments are made from)."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    d = {}
    if kind == "one_pop":
        d["nu"], d["T"] = rng.uniform(0.5, 3), rng.uniform(0.05, 0.07)
        d["gamma"] = rng.uniform(-5, 5)
        d["xx"] = _grid(case["pts"])
        d["phi"] = _phi_1d(d["xx"], 0.0)
    elif kind == "split_mig":
        d["params"] = (rng.uniform(0.5, 3), rng.uniform(0.4, 0.6), rng.uniform(0.18, 0.22),
                       rng.uniform(0.5, 2))
    elif kind == "im":
        d["params"] = (rng.uniform(0.3, 0.7), rng.uniform(0.5, 4), rng.uniform(0.5, 4),
                       rng.uniform(0.1, 0.12), rng.uniform(0.5, 4), rng.uniform(2, 4))
    elif kind in ("batch", "grad"):
        d["params"] = _im_sets(rng, case["n"])
        d["data"] = _counts(rng, case["ns"], 2)
    elif kind == "dfe":
        d["params"] = (rng.uniform(0.3, 0.7), rng.uniform(0.5, 3), rng.uniform(0.5, 3),
                       rng.uniform(0.04, 0.05), rng.uniform(0.5, 2), rng.uniform(0.5, 2))
        d["g"] = -np.logspace(np.log10(case["gmax"]), -3, case["gammas"])
    elif kind in ("growth3", "grad_nd"):
        d["theta"] = _growth3_sets(rng, case.get("n", 1))
        d["data"] = _counts(rng, case["ns"], 3)
    elif kind == "model_batch":
        n = case["n"]
        if case["model"] == "four":
            p = np.array(models.FOUR_DEFAULT)
            d["sets"] = [tuple(float(v) for v in p * f)
                         for f in np.exp(rng.uniform(np.log(0.6), np.log(1.6), (n, 6)))]
        else:
            d["sets"] = [_growth3_params([float(v) for v in th]) for th in _growth3_sets(rng, n)]
        d["data"] = _counts(rng, case["ns"], 4 if case["model"] == "four" else 3)
    return d


def prepare(case, seed):
    kind = case["kind"]
    s = _inputs(case, seed)
    s["case"] = case
    s["pts_l"] = _grids(case)
    if kind in ("batch", "grad"):
        eng = batch.Batch2D(s["pts_l"], (case["ns"],) * 2)
        if case.get("mode") == "per_grid":
            eng.launch_mode, eng.gam_placement = "per_grid", 2
        s["eng"] = eng
    elif kind == "grad_nd":
        s["eng"] = adjoint_nd.Growth3(s["pts_l"], (case["ns"],) * 3)
    elif kind == "model_batch":
        ndim = 4 if case["model"] == "four" else 3
        s["eng"] = batchnd.ModelBatch(case["model"], s["pts_l"], (case["ns"],) * ndim)
    if "data" in s:
        s["data"] = torch.from_numpy(s["data"]).cuda()
    return s


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "one_pop":
        return integration.one_pop(s["phi"], s["xx"], s["T"], s["nu"], gamma=s["gamma"])
    if kind in ("split_mig", "im"):
        f = numerics.make_extrap_func(models.split_mig if kind == "split_mig" else models.IM)
        # (the masked corners are no output)
        return np.ma.filled(f(s["params"], (case["ns"],) * 2, s["pts_l"]), 0.0)
    if kind == "batch":
        was = integration.use_delj_trick
        integration.use_delj_trick = case["delj"]
        try:
            return s["eng"].run(s["params"], data=s["data"], scale=5e3)
        finally:
            integration.use_delj_trick = was
    if kind == "dfe":
        pairs = [(a, b) for a in s["g"] for b in s["g"]]
        return np.stack(dfe.im_sel_spectra(s["params"], (case["ns"],) * 2, s["pts_l"], pairs))
    if kind == "grad":
        return s["eng"].loglik_and_grad(s["params"], s["data"], scale=5e3)
    if kind == "growth3":
        fs = models.growth3(_growth3_params([float(v) for v in s["theta"][0]]),
                            (case["ns"],) * 3, case["pts"])
        return np.ma.filled(fs, 0.0)
    if kind == "model_batch":
        return s["eng"].run(s["sets"], data=s["data"], scale=5e3)
    res = s["eng"].loglik_and_grad_batch(s["theta"], s["data"], scale=5e3)
    return [torch.stack([r[k] for r in res]) for k in range(3)]


# ------------------------------------------------------------------- work

def _schedules(case, d):
    """Per integration of a case, (number of populations, T, sizes(t), migration matrix,
    gammas): what the time loop and the exact values go by."""
    kind = case["kind"]
    if kind == "one_pop":
        return [(1, d["T"], lambda t: (d["nu"],), np.zeros((1, 1)), (d["gamma"],))]
    if kind == "split_mig":
        nu1, nu2, T, m = d["params"]
        return [(2, T, lambda t: (nu1, nu2), np.array([[0, m], [m, 0]]), (0.0, 0.0))]

    def im(p, g=(0.0, 0.0)):
        s, nu1, nu2, T, m12, m21 = (float(v) for v in p)
        return (2, T, lambda t: (s * (nu1 / s) ** (t / T), (1 - s) * (nu2 / (1 - s)) ** (t / T)),
                np.array([[0, m12], [m21, 0]]), g)
    if kind == "im":
        return [im(d["params"])]
    if kind in ("batch", "grad"):
        return [im(p) for p in d["params"]]
    if kind == "dfe":
        return [im(d["params"], (a, b)) for a in d["g"] for b in d["g"]]

    def growth(th):
        a, b, (m12, m13, m23), T = th[0:3], th[3:6], th[6:9], float(th[9])
        return (3, T, lambda t: tuple(u * math.exp(math.log(v / u) * t / T) for u, v in zip(a, b)),
                np.array([[0, m12, m13], [m12, 0, m23], [m13, m23, 0]]), models.GROWTH3_DEFAULT[3])
    if kind in ("growth3", "grad_nd"):
        return [growth([float(v) for v in th]) for th in d["theta"]]
    if case["model"] == "growth3":
        return [growth(list(p[0]) + list(p[1]) + list(p[2]) + [p[4]]) for p in d["sets"]]
    return [(4, p[5], lambda t, p=p: p[:4], p[4] * (1 - np.eye(4)), (0.0,) * 4)
            for p in d["sets"]]


def _dt(nu, m, g):
    """dadi's step from the current sizes, migration and (additive) selection."""
    return min(1e-3 / max(0.25 / nu[k], m[k].sum(), abs(g[k]) * 2 * 0.125)
               for k in range(len(nu)))


def _steps(sched):
    P, T, sizes, m, g = sched
    t, out = 0.0, []
    while t < T:
        step = min(_dt(sizes(t), m, g), T - t)
        t = t + step
        out.append((step, sizes(t)))
    return out


def work(case):
    d = _inputs(case, 0)
    scheds = _schedules(case, d)
    P = scheds[0][0]
    if case["kind"] in ("batch", "grad"):
        steps = int(batch.count_steps(batch.im_instances(d["params"])).sum())
    else:
        steps = sum(len(_steps(s)) for s in scheds)
    points = sum(L ** P for L in _grids(case))
    ns = case.get("ns", 0)
    out = 8 * (points if case["kind"] == "one_pop" else len(scheds) * (ns + 1) ** P)
    flops = POINT_FLOPS * steps * P * points
    # spectra: two multiply-adds per density value and entry of the first contraction
    flops += 4 * len(scheds) * points * (ns + 1)
    if case["kind"] in ("grad", "grad_nd"):
        # the transposed solves, and five sums of two to four operations over the points
        flops = 2 * flops + 15 * steps * P * points
    return {"bytes": 8 * points + out, "flops": flops}


# ------------------------------------------------------------ exact values

def _grid(pts):
    g = 1. / (1. + np.exp(-8. * np.linspace(-1, 1, pts)))
    return (g - g[0]) / (g[-1] - g[0])


def _phi_1d(xx, gamma):
    """Equilibrium density of one population under additive selection."""
    phi = np.empty(len(xx))
    x = xx[1:-1]
    if gamma == 0:
        phi[1:] = 1 / xx[1:]
    else:
        phi[1:-1] = 1 / (x * (1 - x)) * (1 - np.exp(-2 * gamma * (1 - x))) / (1 - np.exp(-2 * gamma))
        phi[-1] = 2 * gamma * np.exp(2 * gamma) / (np.exp(2 * gamma) - 1)
    phi[0] = phi[1]
    return phi


def _split(xx, phi):
    """The last population in two: its mass on the diagonal."""
    L = len(xx)
    out = np.zeros(phi.shape + (L,))
    i = np.arange(1, L - 1)
    out[..., i, i] = phi[..., 1:-1] * 2 / (xx[2:] - xx[:-2])
    return out


def _sweep(phi, xx, ax, dt, nu, m, gamma, delj):
    """One implicit step of every integration along one axis: phi is (n, L, ..., L); dt, nu,
    m (n, P) and gamma are arrays over the integrations."""
    n, P, L = phi.shape[0], phi.ndim - 1, len(xx)
    col = (slice(None),) + (None,) * (P - 1)
    dx, mid = np.diff(xx), (xx[1:] + xx[:-1]) / 2
    df = 2 / np.concatenate([[dx[0]], dx[1:] + dx[:-1], [dx[-1]]])
    d = np.moveaxis(phi, 1 + ax, 0) / dt[col]
    others = [k for k in range(P) if k != ax]
    grids = np.meshgrid(*[xx] * (P - 1), indexing="ij") if P > 1 else []
    flow = sum((m[:, k][col] * g for k, g in zip(others, grids)), np.zeros((n,) + (L,) * (P - 1)))
    total = m[:, others].sum(axis=1)[col]
    sel = lambda x: gamma[col] * x * (1 - x)  # additive: 2 h = 1
    var = lambda x: x * (1 - x) / nu[col]
    M = [flow - total * x + sel(x) for x in mid]
    a, b, c = [np.zeros_like(d) for _ in range(3)]
    b += 1 / dt[col]
    for i in range(L - 1):
        w = 0.5
        if delj:
            wj = 2 * M[i] * dx[i]
            e = np.exp(wj / var(mid[i]))
            w = np.where((e != 1) & (wj != 0), (-e * wj + e * var(mid[i]) - var(mid[i]))
                         / np.where((e != 1) & (wj != 0), wj - e * wj, 1), 0.5)
        up, dn = M[i] * w + var(xx[i]) / (2 * dx[i]), M[i] * (1 - w) - var(xx[i + 1]) / (2 * dx[i])
        a[i + 1] = -df[i + 1] * up
        c[i] = df[i] * dn
        b[i] += df[i] * up
        b[i + 1] -= df[i + 1] * dn
    lo, hi = (slice(None),) + (0,) * (P - 1), (slice(None),) + (L - 1,) * (P - 1)
    m0, m1 = (flow - total * xx[0] + sel(xx[0]))[lo], (flow - total * xx[-1] + sel(xx[-1]))[hi]
    b[0][lo] += np.where(m0 <= 0, (0.5 / nu - m0) * 2 / dx[0], 0)
    b[-1][hi] += np.where(m1 >= 0, (0.5 / nu + m1) * 2 / dx[-1], 0)
    for i in range(1, L):
        r = a[i] / b[i - 1]
        b[i] -= r * c[i - 1]
        d[i] -= r * d[i - 1]
    d[-1] /= b[-1]
    for i in range(L - 2, -1, -1):
        d[i] = (d[i] - c[i] * d[i + 1]) / b[i]
    return np.moveaxis(d, 0, 1 + ax)


def _integrate(phi, xx, scheds, delj):
    """Every integration's density after its time loop; phi is (n, L, ..., L)."""
    P = phi.ndim - 1
    walks = [_steps(s) for s in scheds]
    order = np.argsort([-len(w) for w in walks], kind="stable")
    m = np.array([scheds[k][3] for k in order], dtype=float)
    g = np.array([scheds[k][4] for k in order], dtype=float)
    u = phi[order].copy()
    for t in range(len(walks[order[0]])):
        n = sum(len(walks[k]) > t for k in order)
        dt = np.array([walks[k][t][0] for k in order[:n]])
        nu = np.array([walks[k][t][1] for k in order[:n]], dtype=float)
        add = dt / xx[1] / 2 * 2 ** P / ((xx[2] - xx[0]) * xx[1] ** (P - 1))
        for k in range(P):
            u[(slice(0, n),) + tuple(int(j == k) for j in range(P))] += add
        for k in range(P):
            u[:n] = _sweep(u[:n], xx, k, dt, nu[:, k], m[:n, k], g[:n, k], delj)
    out = np.empty_like(u)
    out[order] = u
    return out


def _tails(n, first, x):
    """I_x(a, n + 1 - a) for a = first .. n: the upper tails of Binomial(n, x)."""
    p = np.array([math.comb(n, j) * x ** j * (1 - x) ** (n - j) for j in range(n + 1)])
    return np.cumsum(p[::-1], axis=0)[::-1][first:]


def _spectrum(phi, ns, xx):
    """Expected spectra of (n, L, ..., L) densities taken as piecewise linear."""
    one = np.diff(_tails(ns + 1, 1, xx), axis=1) / (ns + 1)
    two = np.diff(_tails(ns + 2, 2, xx), axis=1) * (np.arange(1, ns + 2) / ((ns + 1) * (ns + 2)))[:, None]
    for _ in range(phi.ndim - 1):
        slope = np.diff(phi, axis=-1) / np.diff(xx)
        phi = (phi[..., :-1] - slope * xx[:-1]) @ one.T + slope @ two.T
        phi = np.moveaxis(phi, -1, 1)  # the axes come round to their places
    return phi


def _extrapolated(fs, x):
    if len(fs) == 1:
        return fs[0]
    w = [x[1] * x[2] / ((x[0] - x[1]) * (x[0] - x[2])), x[0] * x[2] / ((x[1] - x[0]) * (x[1] - x[2])),
         x[0] * x[1] / ((x[2] - x[0]) * (x[2] - x[1]))]
    ex = sum(a * f for a, f in zip(w, fs))
    with np.errstate(all="ignore"):
        return np.where(np.abs(np.log10(ex / fs[int(np.argmin(x))])) > 10, fs[int(np.argmin(x))], ex)


def _poisson(fs, data, scale):
    model = (scale * fs).reshape(len(fs), -1)
    D = data.reshape(-1)
    ok = (model > 0) & (np.arange(D.size) % (D.size - 1) != 0)
    lg = torch.lgamma(torch.from_numpy(D + 1.0)).numpy()
    t = -model + D * np.log(np.where(ok, model, 1)) - lg
    return np.where(ok, t, 0).sum(axis=1)


def exact(case, seed):
    kind = case["kind"]
    if work(case)["flops"] > 2e10:
        return None
    d = _inputs(case, seed)
    scheds = _schedules(case, d)
    P = scheds[0][0]
    most = max(len(_steps(s)) for s in scheds)
    points = sum(L ** P for L in _grids(case))
    delj = bool(case.get("delj"))
    steps = sum(len(_steps(s)) for s in scheds)
    # about 60 us of array calls per grid row and sweep, and 50 ns per point
    if most * P * sum(_grids(case)) * 6e-5 + steps * P * points * (2e-7 if delj else 5e-8) > 16:
        return None
    if kind == "one_pop":
        return _integrate(d["phi"][None], d["xx"], scheds, False)[0]
    fs, xs = [], []
    for L in _grids(case):
        xx = _grid(L)
        phi = np.stack([_phi_1d(xx, g[0] if kind == "dfe" else 0.0) for *_, g in scheds])
        for _ in range(P - 1):
            phi = np.stack([_split(xx, p) for p in phi])
        fs.append(_spectrum(_integrate(phi, xx, scheds, delj), case["ns"], xx))
        xs.append(xx[1])
    fs = _extrapolated(fs, xs)
    if kind in ("split_mig", "im", "growth3"):
        fs[0].flat[0] = fs[0].flat[-1] = 0
        return fs[0]
    if kind == "dfe":
        return fs
    ll = _poisson(fs, d["data"], 5e3)
    if kind == "batch" or kind == "model_batch":
        return fs, ll, None
    if kind == "grad":
        return ll, None, None
    return [ll, None, fs]
