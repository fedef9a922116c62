"""Cox fits whose events lie unevenly among the rows, against the FP64 oracle:
everybody censored at the end of a fixed follow-up, a handful of events, events
on one side only, few distinct event times, and leading rows without weight (risk
sets that are empty until the first weighted row).  Columns of every row and of
most rows put long runs of one event group into a thread's hands."""
import numpy as np
import pytest

from conftest import assert_contract
from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu

K = 4200


def _problem(kind, strata=0):
    rng = np.random.default_rng(17)
    x = rng.normal(size=K)
    t = rng.exponential(1.0, K) * np.exp(-0.4 * x)
    s = np.sort(rng.integers(0, strata, K)) if strata else np.zeros(K, int)
    if kind == "end":                                  # follow-up ends before most have their event
        limit = np.quantile(t, 0.1)
        y = (t < limit).astype(float)
        t = np.where(y == 1, np.ceil(t / limit * 180) / 180, 2.0)
    elif kind == "rare":
        y = np.zeros(K)
        y[rng.choice(K, 6 * max(1, strata), replace=False)] = 1.0
    elif kind == "late":                               # events among the longest times only: no slot for the rest
        y = (t > np.quantile(t, 0.7)).astype(float)
    elif kind == "ties":                               # visits at four times
        t = np.ceil(np.minimum(t, 3.5))
        y = (rng.random(K) < 0.4).astype(float)
    o = np.lexsort((y, -t, s))
    s, t, y, x = s[o], t[o], y[o], x[o]
    b = D.ColumnBuilder(K).dense(x)
    for n in (50, 900, K - 1):
        b.sparse(np.sort(rng.choice(K, n, replace=False)), rng.normal(size=n))
    for n in (40, 500, 2000, K - 300):
        b.indicator(rng.choice(K, n, replace=False))
    return b.build(D.COX, y, pid=s.astype(np.int32), time=t)


@pytest.mark.parametrize("shape", [None, "1,128", "3,256", "16,512", "16,128"])
@pytest.mark.parametrize("strata", [0, 5])
@pytest.mark.parametrize("kind", ["end", "rare", "late", "ties"])
def test_uneven_events_match_oracle(cuda_lib, monkeypatch, shape, strata, kind):
    from cyclops_b200 import api
    from oracle import oracle as O
    if shape:
        monkeypatch.setenv("CYC_COX_CLUSTER", shape)
    data = _problem(kind, strata)
    rng = np.random.default_rng(2)
    w = rng.integers(0, 3, K).astype(float)
    w[:150] = 0.0                                      # nobody at risk yet
    for weights in (None, w):
        for prior, name in ((D.PRIOR_LAPLACE, "laplace"), (D.PRIOR_NORMAL, "normal")):
            want = O.port().fit(data, prior, 0.4, control=O.make_control(tolerance=1e-7), weights=weights)
            assert want.return_flag == 0
            ctl = api.create_control(tolerance=1e-7)
            fit = api.fit_cyclops_model(data, api.create_prior(name, variance=0.4), ctl, weights=weights)
            assert_contract(fit, want, what=(kind, shape, strata, name, weights is None))
            two = api.batch_fit(data, api.create_prior(name), [0.4, 0.4], [weights, None], ctl)
            assert_contract(two[0], want, what=("batch", kind, shape, strata, name, weights is None))
