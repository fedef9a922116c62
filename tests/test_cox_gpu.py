"""The persistent Cox kernel (csrc/cox.cu) against the FP64 oracle at the sizes
where its parts meet: CTAs and threads without events, columns around its
entries a CTA, strata that end inside or go on past a CTA, ties, zero weights,
rows after the last event, and each place the per-slot arrays may live."""
import numpy as np
import pytest

from conftest import assert_contract
from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


def _problem(K, strata, seed, ties=True, events=0.3, dense=True):
    rng = np.random.default_rng(seed)
    s = np.sort(rng.integers(0, strata, K)) if strata else np.zeros(K, int)
    t = rng.exponential(1.0, K)
    t = np.round(t, 2) + 0.01 if ties else t
    y = (rng.random(K) < events).astype(float)
    if strata > 3:
        y[s == 1] = 0.0                                     # a stratum without events
    y[t <= np.quantile(t, 0.05)] = 0.0                      # rows after the last event (times fall)
    o = np.lexsort((y, -t, s))
    s, t, y = s[o], t[o], y[o]
    b = D.ColumnBuilder(K)
    if dense:
        b.dense(rng.normal(size=K))
    sizes = [n for n in (0, 1, 33, 95, 96, 97, 480, 481, K // 2, K) if n <= K]
    for n in sizes:
        b.sparse(np.sort(rng.choice(K, size=n, replace=False)), rng.normal(size=n))
    for n in sizes[:-1]:
        b.indicator(rng.choice(K, size=n, replace=False))
    return b.build(D.COX, y, pid=s.astype(np.int32), time=t)


def _oracle(data, prior, variance, weights=None, **kw):
    from oracle import oracle as O
    return O.port().fit(data, prior, variance, control=O.make_control(**kw), weights=weights)


@pytest.mark.parametrize("shape", ["1,128", "2,256", "3,128", "8,128", "16,512"])
@pytest.mark.parametrize("strata", [0, 2, 40])
@pytest.mark.parametrize("K", [60, 2100])
def test_shapes_match_oracle(cuda_lib, monkeypatch, shape, strata, K):
    from cyclops_b200 import api
    monkeypatch.setenv("CYC_COX_CLUSTER", shape)
    data = _problem(K, strata, seed=K + strata, ties=strata != 2)
    rng = np.random.default_rng(5)
    w = rng.integers(0, 3, K).astype(float)
    if strata == 40:
        w[data.strata() == 3] = 0.0                         # a stratum without weight
    for weights in (None, w):
        for prior, name in ((D.PRIOR_LAPLACE, "laplace"), (D.PRIOR_NORMAL, "normal")):
            fit = api.fit_cyclops_model(data, api.create_prior(name, variance=0.3), weights=weights)
            want = _oracle(data, prior, 0.3, weights)
            if name == "normal":
                # nothing thresholds: a coefficient whose gradient is 0 in exact
                # arithmetic (an event alone at risk) is 0 to the contract's 1e-9
                for r in (fit, want):
                    r.beta[np.abs(r.beta) < 1e-12] = 0.0
            assert_contract(fit, want, what=(shape, strata, K, name, weights is None))


@pytest.mark.parametrize("K", [30_000, 60_000])
@pytest.mark.parametrize("strata", [0, 7])
def test_slots_beyond_shared_memory(cuda_lib, monkeypatch, K, strata):
    """About 9,000 and 18,000 event groups in one CTA: S1 and S2 alone in
    shared memory, then nothing."""
    from cyclops_b200 import api
    monkeypatch.setenv("CYC_COX_CLUSTER", "1,512")
    data = _problem(K, strata, seed=11, ties=False, dense=False)
    fit = api.fit_cyclops_model(data, api.create_prior("laplace", variance=0.3),
                                api.create_control(tolerance=1e-4))
    assert_contract(fit, _oracle(data, D.PRIOR_LAPLACE, 0.3, tolerance=1e-4), what=(K, strata))


@pytest.mark.parametrize("conv", [D.CONV_LANGE, D.CONV_MITTAL, D.CONV_ONE_STEP, D.CONV_ZHANG_OLES])
@pytest.mark.parametrize("shape", ["1,128", "4,128"])
def test_convergence_rules_match_oracle(cuda_lib, monkeypatch, shape, conv):
    from cyclops_b200 import api
    monkeypatch.setenv("CYC_COX_CLUSTER", shape)
    data = _problem(900, 3, seed=2)
    fit = api.fit_cyclops_model(data, api.create_prior("laplace", variance=0.3),
                                api.create_control(tolerance=1e-4, convergence_type=conv, max_iterations=500))
    assert_contract(fit, _oracle(data, D.PRIOR_LAPLACE, 0.3, tolerance=1e-4, convergence_type=conv,
                                 max_iterations=500), what=(shape, conv))


def test_no_events(cuda_lib):
    from cyclops_b200 import api
    data = _problem(300, 2, seed=4, events=0.0)
    fit = api.fit_cyclops_model(data, api.create_prior("laplace", variance=0.3))
    assert_contract(fit, _oracle(data, D.PRIOR_LAPLACE, 0.3))
