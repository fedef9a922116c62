"""The workloads whose speed is tracked: what users of this framework run,
through its public Python API.

A case is a plain dict.  ``listed()`` gives the fixed ones, ``draw(rng)`` one
more of the same ranges, ``prepare(case, seed)`` the inputs and handles a
program has in hand before the call (the uploaded dataset, prior, control,
fold ids), ``run(state)`` one call, ``work(case)`` the bytes and operations
one call cannot do without, ``exact(case, seed)`` the same outputs from a
plain NumPy restatement in 64 bits.

Kinds of case:

  sweep   the per-coordinate engine as the C++ adapter drives it: linear
          predictor from coefficients, statistics, then gradient / Hessian
          and update of a few columns, one call each
  fit     fit_cyclops_model: one regularised fit to convergence
  auto    cv_auto_search: the default cross-validation (10 folds a step)
  grid    cv_grid_fit: folds x a grid of prior variances
  boot    batch_fit on bootstrap replicate weights
  fisher  asymptotic_variance at given coefficients (standard errors)

All data are seeded and synthetic: indicator covariates with a uniform or a
Zipf(1.1) column frequency (claims data), or sparse real-valued ones; the
sizes follow the benchmark's configurations and the tests, scaled so that a
call takes at most about two seconds.
"""
import math

import numpy as np
import torch

from cyclops_b200 import api
from cyclops_b200 import data as D

_MODELS = {"lr": D.LR, "pr": D.PR, "clr": D.CLR, "cpr": D.CPR, "cox": D.COX}
_KINDS = ("sweep", "fit", "auto", "grid", "boot", "fisher")


def _case(name, kind, model, rows, columns, per_column, **more):
    c = {"kind": kind, "model": model, "rows": rows, "columns": columns, "per_column": per_column,
         "zipf": 0.0, "real": False, "dense": 0, "offset": False, "strata": 0, "prior": "laplace",
         "variance": 200.0, "weighted": False, "swindle": False, "sweep": 0, "folds": 0, "grid": 0, "fits": 0}
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest calls: one engine call per virtual of the reference's
        # engine interface, 24 columns of the 10k x 1k logistic problem
        _case("sweep_lr", "sweep", "lr", 10_000, 1_000, 100, sweep=24),
        # the plain fit: 10k x 1k indicators at 1 %, Laplace lambda 0.1
        _case("fit_lr", "fit", "lr", 10_000, 1_000, 100),
        # a larger claims-like design under a strong penalty with the
        # reference's active-set passes
        _case("fit_lr_swindle", "fit", "lr", 200_003, 1_200, 700, zipf=1.1, variance=0.02, swindle=True),
        # Poisson rates: offset, dense covariates, Zipf indicators, normal prior
        _case("fit_pr", "fit", "pr", 100_003, 600, 1_500, zipf=1.1, dense=3, offset=True, prior="normal",
              variance=1.0),
        # matched case-control sets, 1:4
        _case("fit_clr", "fit", "clr", 20_000, 500, 200, strata=4_000),
        # survival, tied strata-free cohort with real-valued covariates
        _case("fit_cox", "fit", "cox", 20_011, 500, 200, real=True),
        # a large stratified survival cohort, weighted
        _case("fit_cox_strata", "fit", "cox", 500_009, 250, 500, strata=100, weighted=True),
        # the default cross-validation: ten folds a step until it settles
        _case("auto_lr", "auto", "lr", 10_007, 400, 100, folds=10),
        # the largest: a CV grid over half a million rows, 200 fits
        _case("grid_lr", "grid", "lr", 500_000, 4_000, 1_000, zipf=1.1, folds=10, grid=20),
        # cross-validated Cox, each fold with its own risk sets
        _case("grid_cox", "grid", "cox", 30_000, 120, 300, folds=10, grid=2),
        # bootstrap replicates of a Poisson fit
        _case("boot_pr", "boot", "pr", 50_003, 300, 400, zipf=1.1, variance=1.0, fits=24),
        # standard errors of 200 coefficients
        _case("fisher_lr", "fisher", "lr", 50_000, 200, 1_000, zipf=1.1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("sweep", "fit", "fit", "fit", "cox", "auto", "grid", "boot", "fisher"))
    z = rng.choice((0.0, 1.1))
    if kind == "sweep":
        model = rng.choice(("lr", "pr", "clr", "cox"))
        rows = _log(rng, 1_000, 200_000)
        return _case(None, "sweep", model, rows, _log(rng, 60, 1_000), max(10, rows // rng.randint(20, 400)),
                     sweep=rng.randint(8, 48), zipf=z, strata=rows // 5 if model == "clr" else 0,
                     real=rng.random() < 0.4)
    if kind == "fit":
        model = rng.choice(("lr", "lr", "pr", "clr", "cpr"))
        rows = _log(rng, 2_000, 200_000)
        grouped = model in ("clr", "cpr")
        prior = rng.choice(("laplace", "normal"))
        swindle = model == "lr" and prior == "laplace" and rng.random() < 0.4
        return _case(None, "fit", model, rows, _log(rng, 50, 600), max(40, rows // rng.randint(60, 200)), zipf=z,
                     real=rng.random() < 0.3, dense=0 if grouped else rng.choice((0, 1, 4)),
                     offset=model == "pr" and rng.random() < 0.5, strata=rows // rng.randint(4, 10) if grouped else 0,
                     prior=prior, variance=0.05 if swindle else math.exp(rng.uniform(-2.0, 2.0)),
                     weighted=rng.random() < 0.3, swindle=swindle)
    if kind == "cox":
        rows = _log(rng, 5_000, 500_000)
        return _case(None, "fit", "cox", rows, _log(rng, 40, 250), max(30, rows // rng.randint(50, 1_000)),
                     real=rng.random() < 0.5, strata=rng.choice((0, 0, 30, rows // 200)),
                     variance=math.exp(rng.uniform(0.0, 5.0)), weighted=rng.random() < 0.3)
    if kind == "auto":
        model = rng.choice(("lr", "pr"))
        rows = _log(rng, 4_000, 40_000)
        return _case(None, "auto", model, rows, _log(rng, 40, 300), max(40, rows // rng.randint(50, 120)), zipf=z,
                     folds=rng.choice((5, 10)))
    if kind == "grid":
        model = rng.choice(("lr", "lr", "pr", "cox"))
        if model == "cox":
            return _case(None, "grid", "cox", _log(rng, 5_000, 60_000), _log(rng, 40, 120), 300, folds=5,
                         grid=rng.randint(1, 3), real=rng.random() < 0.5)
        rows = _log(rng, 10_000, 400_000)
        return _case(None, "grid", model, rows, _log(rng, 80, 600), max(50, rows // rng.randint(100, 500)), zipf=z,
                     folds=rng.choice((5, 10)), grid=rng.randint(2, 16))
    if kind == "boot":
        rows = _log(rng, 5_000, 100_000)
        return _case(None, "boot", rng.choice(("lr", "pr")), rows, _log(rng, 60, 400),
                     max(40, rows // rng.randint(60, 200)), zipf=z, real=rng.random() < 0.3,
                     variance=math.exp(rng.uniform(-1.0, 1.0)), fits=rng.randint(5, 40))
    model = rng.choice(("lr", "pr", "clr"))
    rows = _log(rng, 5_000, 100_000)
    return _case(None, "fisher", model, rows, _log(rng, 20, 250), max(50, rows // rng.randint(20, 100)), zipf=z,
                 real=rng.random() < 0.3, strata=rows // 5 if model == "clr" else 0)


# ---- data ---------------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _problem(case, seed):
    """The host arrays of one seeded problem (column order and row order as
    the reference ingests them)."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 1_000_003 + 12_345)
    rng = np.random.default_rng([int(seed), 77])
    K, P, S = case["rows"], case["columns"], case["strata"]
    model = _MODELS[case["model"]]
    # column sizes, then distinct rows of each column
    total = case["per_column"] * P
    if case["zipf"]:
        w = np.arange(1, P + 1, dtype=np.float64) ** -case["zipf"]
        counts = np.minimum(w / w.sum() * total, 0.4 * K)
        counts = np.maximum(20, np.minimum(counts * (total / counts.sum()), 0.4 * K)).astype(np.int64)
    else:
        counts = np.maximum(5, rng.binomial(K, min(0.5, case["per_column"] / K), size=P))
    cols = torch.repeat_interleave(torch.arange(P, device=dev), torch.as_tensor(counts, device=dev))
    rows = torch.randint(0, K, (int(counts.sum()),), generator=gen, device=dev)
    keys = torch.unique(cols * K + rows)
    cols, rows = keys // K, keys % K
    x = torch.randn(rows.shape[0], generator=gen, device=dev, dtype=torch.float64) if case["real"] else None
    beta = torch.zeros(P, dtype=torch.float64)
    true = torch.as_tensor(rng.choice(P, size=min(50, P), replace=False))
    beta[true] = torch.as_tensor(rng.normal(0.0, 0.4, size=true.shape[0]))
    contrib = beta.to(dev)[cols] * (x if x is not None else 1.0)
    eta = torch.zeros(K, dtype=torch.float64, device=dev).index_add_(0, rows, contrib)
    eta = eta.cpu().numpy()
    dense = rng.normal(0.0, 1.0, size=(case["dense"], K))
    if case["dense"]:
        eta = eta + 0.2 * dense.sum(axis=0)
    pid = time = None
    order = None
    if model == D.LR:
        y = (rng.random(K) < 1.0 / (1.0 + np.exp(2.0 - eta))).astype(np.float64)
    elif model == D.PR:
        if case["offset"]:
            time = np.log(rng.exponential(1.0, size=K) + 0.05)
            eta = eta + time
        y = rng.poisson(np.exp(np.clip(eta - 1.0, -30.0, 4.0))).astype(np.float64)
    elif model in (D.CLR, D.CPR):
        pid = np.sort(np.concatenate([np.arange(S), rng.integers(0, S, size=K - S)])).astype(np.int32)
        if model == D.CPR:
            y = rng.poisson(np.exp(np.clip(eta - 0.5, -30.0, 4.0))).astype(np.float64)
        else:
            # one case a stratum, drawn in proportion to exp(eta)
            score = eta + rng.gumbel(size=K)
            best = np.lexsort((score, pid))
            last = np.append(np.flatnonzero(np.diff(pid)), K - 1)
            y = np.zeros(K)
            y[best[last]] = 1.0
    else:
        t = rng.exponential(1.0, size=K) / np.exp(eta)
        t = np.round(t ** (1.0 / 1.2), 5) + 1e-5
        y = (rng.random(K) >= 0.7).astype(np.float64)
        s = rng.integers(0, S, size=K) if S else np.zeros(K, np.int64)
        order = np.lexsort((y, -t, s))
        y, time, pid = y[order], t[order], s[order].astype(np.int32)
        inv = np.empty(K, np.int64)
        inv[order] = np.arange(K)
        rows = torch.as_tensor(inv, device=dev)[rows]
        keys, at = torch.sort(cols * K + rows)
        cols, rows = keys // K, keys % K
        x = x[at] if x is not None else None
    n = torch.bincount(cols, minlength=P).cpu().numpy()
    rows, x = rows.to(torch.int32).cpu().numpy(), x.cpu().numpy() if x is not None else None
    # an offset, then the intercept and the dense columns, then the others
    lead = []
    intercept = model in (D.LR, D.PR)
    if case["offset"]:
        lead.append(time)
    if intercept:
        lead.append(np.ones(K))
    lead.extend(dense)
    J = len(lead) + P
    fmt = np.full(J, D.SPARSE if case["real"] else D.INDICATOR, np.int32)
    fmt[:len(lead)] = D.DENSE
    col_ptr = np.concatenate([np.zeros(len(lead) + 1, np.int64), np.cumsum(n)])
    lens = np.concatenate([np.full(len(lead), K, np.int64), n if case["real"] else np.zeros(P, np.int64)])
    val_ptr = np.concatenate([np.zeros(1, np.int64), np.cumsum(lens)])
    val = np.concatenate(lead + ([x] if x is not None else [])) if lead or x is not None else np.zeros(0)
    prob = {"model": model, "K": K, "J": J, "y": y, "pid": pid, "time": time, "fmt": fmt, "col_ptr": col_ptr,
            "col_idx": rows, "val_ptr": val_ptr, "col_val": val, "offset": bool(case["offset"]),
            "intercept": intercept}
    prob["weights"] = rng.integers(1, 4, size=K).astype(np.float64) if case["weighted"] else None
    if case["folds"]:
        prob["fold"] = (rng.permutation(K) % case["folds"]).astype(np.int32)
        lam = np.exp(np.linspace(math.log(0.1), math.log(3.0), max(1, case["grid"])))
        prob["variances"] = 2.0 / lam ** 2
    if case["fits"]:
        prob["boot"] = np.stack([np.bincount(rng.integers(0, K, size=K), minlength=K).astype(np.float64)
                                 for _ in range(case["fits"])])
    if case["kind"] in ("sweep", "fisher"):
        b = rng.normal(0.0, 0.1, size=J)
        if case["offset"]:
            b[0] = 1.0
        prob["beta"] = b
        prob["sweep"] = np.sort(rng.choice(J, size=min(case["sweep"], J), replace=False))
        prob["delta"] = rng.normal(0.0, 0.02, size=len(prob["sweep"]))
    return prob


def prepare(case, seed):
    p = _problem(case, seed)
    data = D.CyclopsData(model=p["model"], y=p["y"], col_format=p["fmt"], col_ptr=p["col_ptr"], col_idx=p["col_idx"],
                         val_ptr=p["val_ptr"], col_val=p["col_val"], pid=p["pid"], time=p["time"],
                         has_offset=p["offset"], has_intercept=p["intercept"])
    state = {"kind": case["kind"], "data": api.Dataset(data), "p": p, "folds": case["folds"],
             "prior": api.create_prior(case["prior"], variance=case["variance"]),
             "control": api.create_control(use_kkt_swindle=case["swindle"])}
    if case["kind"] == "sweep":
        state["engine"] = api.Engine(state["data"])
        state["engine"].set_weights(None)
    return state


def run(state):
    kind, ds, p = state["kind"], state["data"], state["p"]
    prior, control = state["prior"], state["control"]
    if kind == "sweep":
        e = state["engine"]
        e.compute_fixed_terms_in_gradient_and_hessian()
        e.compute_xbeta(p["beta"])
        e.compute_remaining_statistics()
        gh = np.zeros((len(p["sweep"]), 2))
        for i, j in enumerate(p["sweep"]):
            e.compute_numerator_for_gradient(int(j))
            gh[i] = e.compute_gradient_and_hessian(int(j))
            e.update_xbeta(float(p["delta"][i]), int(j))
        return {"gh": gh, "objective": e.get_gradient_objective(), "log_likelihood": e.get_log_likelihood(),
                "xbeta": e.get_xbeta()}
    if kind == "fit":
        r = api.fit_cyclops_model(ds, prior, control, weights=p["weights"])
        return {"beta": r.beta, "log_likelihood": r.log_likelihood, "log_prior": r.log_prior,
                "iterations": r.iterations, "flag": r.return_flag}
    if kind == "auto":
        r = api.cv_auto_search(ds, prior, p["fold"], state["folds"], control=control)
        return {"variance": r.variance, "expected": r.expected, "tried": r.tried}
    if kind == "grid":
        r = api.cv_grid_fit(ds, prior, p["fold"], state["folds"], p["variances"], control=control)
        return {"beta": np.stack([f.beta for f in r.fits]), "pred_loglik": r.pred_loglik, "grid_mean": r.grid_mean,
                "log_likelihood": np.array([f.log_likelihood for f in r.fits]),
                "iterations": np.array([f.iterations for f in r.fits])}
    if kind == "boot":
        r = api.batch_fit(ds, prior, [prior.variance] * len(p["boot"]), weights=p["boot"], control=control)
        return {"beta": np.stack([f.beta for f in r]), "log_likelihood": np.array([f.log_likelihood for f in r]),
                "iterations": np.array([f.iterations for f in r])}
    r = api.asymptotic_variance(ds, p["beta"], prior)
    return {"fisher": r.fisher, "standard_errors": r.standard_errors}


# ---- work -----------------------------------------------------------------------

# coordinate cycles a fit of each model takes on such data, to about a factor of two
_CYCLES = {"lr": 25, "pr": 30, "clr": 15, "cpr": 15, "cox": 8}


def work(case):
    """A coordinate reads its column and its rows' state once and, as it
    moves, writes that state once; the data of a fit are passed once a cycle.
    Cox reads and renews the risk-set sums of its events (30 % of the rows)
    at every coordinate."""
    K, P = case["rows"], case["columns"]
    nnz = min(case["per_column"], 0.5 * K) * P
    entry = 4.0 + (8.0 if case["real"] else 0.0)
    dense = (case["dense"] + case["offset"] + (case["model"] in ("lr", "pr"))) * K
    flops = 30.0 * (nnz + dense)
    state = 16.0 * (nnz + dense)
    if case["model"] == "cox":
        state += 16.0 * 0.3 * K * P
        flops += 8.0 * 0.3 * K * P
    columns = entry * nnz + 8.0 * dense
    if case["kind"] == "sweep":
        share = case["sweep"] / P
        return {"bytes": columns * (1.0 + share) + state * share + 40.0 * K, "flops": flops * share + 2.0 * nnz + 30.0 * K}
    if case["kind"] == "fisher":
        return {"bytes": columns + 8.0 * K + 8.0 * P * P, "flops": 2.0 * nnz * P * min(1.0, case["per_column"] / K) + 30.0 * K}
    fits = {"fit": 1, "auto": 8 * case["folds"], "grid": case["folds"] * max(1, case["grid"]), "boot": case["fits"]}[case["kind"]]
    cycles = _CYCLES[case["model"]]
    return {"bytes": cycles * (columns + fits * (state + 16.0 * K)), "flops": cycles * fits * (flops + 3.0 * K)}


# ---- the same results in plain NumPy ----------------------------------------------

def _columns(p):
    out = []
    for j in range(p["J"]):
        rows = None if p["fmt"][j] == D.DENSE else p["col_idx"][p["col_ptr"][j]:p["col_ptr"][j + 1]]
        x = None if p["fmt"][j] == D.INDICATOR else p["col_val"][p["val_ptr"][j]:p["val_ptr"][j + 1]]
        if rows is None:
            rows = np.arange(p["K"])
        out.append((rows, x))
    return out


def _strata(p):
    if p["pid"] is None:
        return np.zeros(p["K"], np.int64)
    return np.concatenate([[0], np.cumsum(p["pid"][1:] != p["pid"][:-1])])


def _risk_groups(p, w):
    """Risk-set group of every row (rows in time order within a stratum):
    tied events share one; rows of weight zero join the group before."""
    s, t, y = _strata(p), p["time"], p["y"]
    on = np.flatnonzero(w != 0)
    new = np.ones(on.size, bool)
    a, b = on[1:], on[:-1]
    new[1:] = ~((s[a] == s[b]) & (y[b] == 1) & (t[a] == t[b]) & (y[a] == y[b]))
    g = np.zeros(p["K"], np.int64)
    g[on] = np.cumsum(new) - 1
    marks = np.zeros(p["K"], np.int64)
    marks[on] = g[on]
    g = np.maximum.accumulate(marks)
    n = int(g.max()) + 1
    first = np.zeros(n, np.int64)
    first[g[on[::-1]]] = s[on[::-1]]
    start = np.concatenate([[True], first[1:] != first[:-1]])
    return g, n, start


def _segmented(v, start):
    """Inclusive sums that restart where `start` is set."""
    c = np.cumsum(v.astype(np.longdouble))
    at = np.flatnonzero(start)
    base = np.zeros(at.size, np.longdouble)
    base[1:] = c[at[1:] - 1]
    return (c - np.repeat(base, np.diff(np.append(at, v.size)))).astype(np.float64)


class _State:
    """The statistics of F fits (columns) under weights w (K, F)."""

    def __init__(self, p, w):
        self.p, self.w, self.m = p, w, p["model"]
        self.cols = _columns(p)
        self.xb = np.zeros(w.shape)
        if self.m == D.COX:
            self.g, self.n, self.start = _risk_groups(p, w[:, 0])
            self.events = np.bincount(self.g, p["y"] * w[:, 0], self.n)
        elif self.m in (D.CLR, D.CPR):
            self.g = _strata(p)
            self.n = int(self.g[-1]) + 1
            self.events = np.stack([np.bincount(self.g, p["y"] * w[:, f], self.n) for f in range(w.shape[1])], axis=1)
        self.xjy = np.stack([((x[:, None] if x is not None else 1.0) * (p["y"][r])[:, None] * w[r]).sum(axis=0)
                             for r, x in self.cols])

    def renew(self):
        if self.m == D.COX:
            self.D = _segmented(np.bincount(self.g, self.w[:, 0] * np.exp(self.xb[:, 0]), self.n), self.start)
        elif self.m in (D.CLR, D.CPR):
            self.D = np.stack([np.bincount(self.g, np.exp(self.xb[:, f]), self.n) for f in range(self.xb.shape[1])], axis=1)

    def gradient(self, j):
        r, x = self.cols[j]
        xx = x[:, None] if x is not None else np.ones((r.size, 1))
        v = self.xb[r]
        if self.m == D.LR:
            q = 1.0 / (1.0 + np.exp(-v))
            g, h = (self.w[r] * q * xx).sum(axis=0), (self.w[r] * q * (1.0 - q) * xx * xx).sum(axis=0)
        elif self.m == D.PR:
            g, h = (self.w[r] * np.exp(v) * xx).sum(axis=0), (self.w[r] * np.exp(v) * xx * xx).sum(axis=0)
        elif self.m == D.COX:
            e = self.w[r, 0] * np.exp(v[:, 0]) * xx[:, 0]
            a = _segmented(np.bincount(self.g[r], e, self.n), self.start)
            b = _segmented(np.bincount(self.g[r], e * xx[:, 0], self.n), self.start)
            t = a / self.D
            g = np.array([(self.events * t).sum()])
            h = np.array([(self.events * (b / self.D - t * t)).sum()])
        else:
            e = np.exp(v) * xx
            s, at = np.unique(self.g[r], return_inverse=True)
            a, b = np.zeros((s.size, v.shape[1])), np.zeros((s.size, v.shape[1]))
            np.add.at(a, at, e)
            np.add.at(b, at, e * xx)
            t = a / self.D[s]
            g, h = (self.events[s] * t).sum(axis=0), (self.events[s] * (b / self.D[s] - t * t)).sum(axis=0)
        if r.size == 0:
            return np.zeros(v.shape[1]), np.zeros(v.shape[1])
        return g - self.xjy[j], h

    def move(self, j, d):
        r, x = self.cols[j]
        old = np.exp(self.xb[r]) if self.m in (D.CLR, D.CPR) else None
        self.xb[r] += d * (x[:, None] if x is not None else 1.0)
        if self.m in (D.CLR, D.CPR):
            np.add.at(self.D, self.g[r], np.exp(self.xb[r]) - old)
        elif self.m == D.COX and np.any(d != 0):
            self.renew()

    def objective(self):
        return (self.xb * self.p["y"][:, None] * self.w).sum(axis=0)

    def log_likelihood(self):
        y, w, xb = self.p["y"][:, None], self.w, self.xb
        if self.m == D.LR:
            return (w * (y * xb - np.log1p(np.exp(xb)))).sum(axis=0)
        if self.m == D.PR:
            fact = -np.array([math.lgamma(v + 1.0) for v in range(int(self.p["y"].max()) + 1)])
            return (w * (y * xb - np.exp(xb) + fact[self.p["y"].astype(int)][:, None])).sum(axis=0)
        ev = self.events if self.m != D.COX else self.events[:, None]
        dd = self.D if self.m != D.COX else self.D[:, None]
        ll = (w * y * xb).sum(axis=0) - np.where(ev != 0, ev * np.log(dd), 0.0).sum(axis=0)
        if self.m == D.CPR:
            fact = -np.array([math.lgamma(v + 1.0) for v in range(int(self.p["y"].max()) + 1)])
            ll = ll + (w * fact[self.p["y"].astype(int)][:, None]).sum(axis=0)
        return ll


def _flat(p, prior):
    """Columns without a prior: the intercept."""
    flat = np.zeros(p["J"], bool)
    if prior != "none" and p["intercept"]:
        flat[1 if p["offset"] else 0] = True
    return flat


def _step(kind, flat, var, b, g, h, bound):
    bad = h < 0
    g, h = np.where(bad, 0.0, g), np.where(bad, 0.0, h)
    with np.errstate(all="ignore"):
        if flat:
            d = -(g / h)
        elif kind == "normal":
            d = -(g + b / var) / (h + 1.0 / var)
        else:
            lam = np.sqrt(2.0 / var)
            neg, pos = -(g - lam) / h, -(g + lam) / h
            zero = np.where(neg < 0, neg, np.where(pos > 0, pos, 0.0))
            d = np.where(b == 0, zero, np.where(b < 0, neg, pos))
            d = np.where((b != 0) & (np.sign(b + d) != np.sign(b)), -b, d)
    d = np.clip(d, -bound, bound)
    return d, np.maximum(np.maximum(2 * np.abs(d), bound / 2), 1e-3)


def _descend(p, st, beta, var, prior, active, cycles=1000, tol=1e-6):
    """Cyclic coordinate descent of the F fits until each one's objective
    settles; beta is changed in place."""
    F = beta.shape[1]
    flat = _flat(p, prior)
    bound = np.full(beta.shape, 2.0)
    last, done, iters = st.objective(), np.zeros(F, bool), np.zeros(F, np.int64)
    for it in range(1, cycles + 1):
        for j in range(p["J"]):
            if not active[j]:
                continue
            g, h = st.gradient(j)
            d, nb = _step(prior, flat[j], var, beta[j], g, h, bound[j])
            d = np.where(done, 0.0, d)
            bound[j] = np.where(done, bound[j], nb)
            beta[j] += d
            if np.any(d != 0):
                st.move(j, d)
        o = st.objective()
        near = np.abs(o - last) / (np.abs(o) + 1.0) < tol
        iters = np.where(done, iters, it)
        last = np.where(done, last, o)
        done |= near
        if done.all():
            break
    return iters


def _log_prior(p, beta, var, prior):
    keep = ~_flat(p, prior)
    b = beta[keep]
    if prior == "normal":
        return (-0.5 * np.log(2.0 * np.pi * var) - 0.5 * b * b / var).sum(axis=0)
    lam = np.sqrt(2.0 / var)
    return (np.log(0.5 * lam) - lam * np.abs(b)).sum(axis=0)


def _fit(p, w, var, case):
    """F fits: beta (J, F), cycles and the final state."""
    st = _State(p, w)
    F = w.shape[1]
    beta = np.zeros((p["J"], F))
    free = np.ones(p["J"], bool)
    if p["offset"]:
        beta[0] = 1.0
        free[0] = False
        st.xb += p["time"][:, None]
    st.renew()
    if not case["swindle"]:
        return beta, _descend(p, st, beta, var, case["prior"], free), st
    flat = _flat(p, case["prior"])
    active = free & flat
    while True:
        iters = _descend(p, st, beta, var, case["prior"], active)
        idle = np.flatnonzero(free & ~active)
        moved = [j for j in idle if abs(st.gradient(j)[0][0]) > math.sqrt(2.0 / var[0])]
        if not moved:
            return beta, iters, st
        active[moved] = True


def _seconds(case):
    """What the restatement takes, roughly, on one core."""
    K, P, F = case["rows"], case["columns"], max(1, case["fits"])
    n = min(case["per_column"], 0.5 * K)
    lead = (case["dense"] + 1) * K
    cycles = 3 * _CYCLES[case["model"]]
    if case["swindle"]:
        cycles *= 2
    if case["kind"] in ("sweep", "fisher"):
        return 1.0
    if case["kind"] == "grid":
        F = case["folds"] * max(1, case["grid"])
    if case["model"] == "cox":
        return F * cycles / 2 * P * (6e-5 + 1.2e-7 * K)
    return cycles * (P * (6e-5 + 4e-8 * n * F) + 4e-8 * lead * F)


def exact(case, seed):
    kind = case["kind"]
    if kind == "auto" or _seconds(case) > 18.0:
        return None          # a search over whole cross-validations, or too long in NumPy
    p = _problem(case, seed)
    K = p["K"]
    if kind == "sweep":
        st = _State(p, np.ones((K, 1)))
        for j, (r, x) in enumerate(st.cols):
            st.xb[r, 0] += p["beta"][j] * (x if x is not None else 1.0)
        st.renew()
        gh = np.zeros((len(p["sweep"]), 2))
        for i, j in enumerate(p["sweep"]):
            g, h = st.gradient(j)
            gh[i] = g[0], h[0]
            st.move(j, np.array([p["delta"][i]]))
        return {"gh": gh, "objective": float(st.objective()[0]), "log_likelihood": float(st.log_likelihood()[0]),
                "xbeta": st.xb[:, 0].copy()}
    if kind == "fisher":
        keep = np.arange(p["J"])
        X = np.zeros((K, p["J"]))
        for j, (r, x) in enumerate(_columns(p)):
            X[r, j] = 1.0 if x is None else x
        xb = X @ p["beta"]
        if p["model"] == D.LR:
            q = 1.0 / (1.0 + np.exp(-xb))
            info = X.T @ (X * (q * (1.0 - q))[:, None])
        elif p["model"] == D.PR:
            info = X.T @ (X * np.exp(xb)[:, None])
        else:
            s = _strata(p)
            e = np.exp(xb)
            q = e / np.bincount(s, e)[s]
            at = np.flatnonzero(np.concatenate([[True], s[1:] != s[:-1]]))
            T = np.add.reduceat(X * q[:, None], at, axis=0)
            info = X.T @ (X * q[:, None]) - T.T @ T
        return {"fisher": info[np.ix_(keep, keep)], "standard_errors": np.sqrt(np.diag(np.linalg.inv(info)))}
    if kind == "fit":
        w = np.ones((K, 1)) if p["weights"] is None else p["weights"][:, None]
        var = np.array([case["variance"]])
        beta, iters, st = _fit(p, w, var, case)
        return {"beta": beta[:, 0].copy(), "log_likelihood": float(st.log_likelihood()[0]),
                "log_prior": float(_log_prior(p, beta, var, case["prior"])[0]), "iterations": None, "flag": None}
    if kind == "boot":
        var = np.full(len(p["boot"]), case["variance"])
        beta, iters, st = _fit(p, np.ascontiguousarray(p["boot"].T), var, case)
        return {"beta": np.ascontiguousarray(beta.T), "log_likelihood": st.log_likelihood(), "iterations": None}
    # grid: fit i = (variance i / folds, fold i % folds)
    F = case["folds"] * len(p["variances"])
    fold = np.arange(F) % case["folds"]
    var = np.repeat(p["variances"], case["folds"])
    w = (p["fold"][:, None] != fold[None, :]).astype(np.float64)
    if p["model"] == D.COX:
        one = [_fit(p, np.ascontiguousarray(w[:, f:f + 1]), var[f:f + 1], case) for f in range(F)]
        return {"beta": np.stack([b[:, 0] for b, _, _ in one]), "pred_loglik": None, "grid_mean": None,
                "log_likelihood": np.array([st.log_likelihood()[0] for _, _, st in one]), "iterations": None}
    beta, iters, st = _fit(p, w, var, case)
    held = (1.0 - w) * p["y"][:, None]
    if p["model"] == D.LR:
        pred = (held * (st.xb - np.log1p(np.exp(st.xb)))).sum(axis=0)
    else:
        pred = held * st.xb - (1.0 - w) * np.exp(st.xb)
        pred = pred.sum(axis=0)
    return {"beta": np.ascontiguousarray(beta.T), "pred_loglik": pred,
            "grid_mean": pred.reshape(-1, case["folds"]).mean(axis=1), "log_likelihood": st.log_likelihood(),
            "iterations": None}
