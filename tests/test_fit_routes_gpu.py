"""The two routes of a single lr, pr, clr or cpr fit -- one cluster for the whole
loop, or the engine's kernels over the whole device a column at a time -- against
the FP64 oracle and one another, and the rule between them."""
import numpy as np
import pytest

from conftest import assert_contract
from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


def _problem(model, K=1300, seed=0):
    """An offset-free design with an empty column, long and short, dense, real and indicator ones."""
    rng = np.random.default_rng(seed + model)
    b = D.ColumnBuilder(K)
    grouped = model in (D.CLR, D.CPR)
    if not grouped:
        b.intercept()
    z = rng.normal(size=K)
    b.dense(z)
    for n in (0, 1, 200, 1200):
        b.sparse(np.sort(rng.choice(K, n, replace=False)), rng.normal(size=n))
    for n in (30, 1024, K - 1):
        b.indicator(rng.choice(K, n, replace=False))
    pid = None
    if grouped:
        pid = np.sort(rng.integers(0, K // 6, K)).astype(np.int32)
        y = (rng.random(K) < 0.3).astype(float) if model == D.CLR else rng.poisson(0.5, K).astype(float)
    elif model == D.LR:
        y = (rng.random(K) < 1 / (1 + np.exp(1 - 0.5 * z))).astype(float)
    else:
        y = rng.poisson(np.exp(0.3 * z - 0.5)).astype(float)
    return b.build(model, y, pid=pid, has_intercept=not grouped)


@pytest.mark.parametrize("route", ["columns", "cluster"])
@pytest.mark.parametrize("conv", [D.CONV_GRADIENT, D.CONV_LANGE, D.CONV_MITTAL, D.CONV_ONE_STEP, D.CONV_ZHANG_OLES])
@pytest.mark.parametrize("model", [D.LR, D.PR, D.CLR, D.CPR])
def test_route_matches_oracle(cuda_lib, monkeypatch, route, conv, model):
    from cyclops_b200 import api
    from oracle import oracle as O
    monkeypatch.setenv("CYC_FIT_ROUTE", route)
    data = _problem(model)
    w = np.random.default_rng(3).integers(0, 3, data.K).astype(float)
    ctl = dict(tolerance=1e-5, convergence_type=conv, max_iterations=300)
    for weights in (None, w):
        for prior, name in ((D.PRIOR_LAPLACE, "laplace"), (D.PRIOR_NORMAL, "normal")):
            want = O.port().fit(data, prior, 0.5, control=O.make_control(**ctl), weights=weights)
            got = api.fit_cyclops_model(data, api.create_prior(name, variance=0.5), api.create_control(**ctl),
                                        weights=weights)
            assert_contract(got, want, what=(route, conv, model, name, weights is None))


@pytest.mark.parametrize("model", [D.LR, D.PR, D.CLR])
def test_routes_agree_beyond_the_plain_fit(cuda_lib, monkeypatch, model):
    """Active-set passes, held coefficients, starting values, profile bounds."""
    from cyclops_b200 import api
    ds = api.Dataset(_problem(model))
    x = 0 if model == D.CLR else 1                     # the dense column
    prior = api.create_prior("laplace", variance=0.05)
    start = np.zeros(ds.data.J)
    start[[x, x + 3]] = (0.2, -0.1)
    out = {}
    for route in ("columns", "cluster"):
        monkeypatch.setenv("CYC_FIT_ROUTE", route)
        flat = api.create_prior("laplace", variance=0.5, exclude=[x])
        b = api.profile_bounds(ds, [x], flat)
        out[route] = (api.fit_cyclops_model(ds, prior, api.create_control(use_kkt_swindle=True)),
                      api.fit_cyclops_model(ds, prior, starting_coefficients=start, fixed_coefficients=[x]), b)
    for a, b in zip(out["columns"][:2], out["cluster"][:2]):
        assert_contract(a, b, what=model)
    np.testing.assert_allclose(out["columns"][2].lower, out["cluster"][2].lower, rtol=1e-5)
    np.testing.assert_allclose(out["columns"][2].upper, out["cluster"][2].upper, rtol=1e-5)


@pytest.mark.parametrize("kind,route", [("long", "columns"), ("short", "cluster")])
def test_rule(cuda_lib, monkeypatch, kind, route):
    """Fits of dense columns over many matched sets run over the device, fits of short columns in a cluster."""
    from cyclops_b200 import api
    rng = np.random.default_rng(5)
    K = 120_000
    b = D.ColumnBuilder(K)
    for _ in range(4):
        if kind == "long":
            b.dense(rng.normal(size=K))
        else:
            b.indicator(rng.choice(K, 300, replace=False))
    data = b.build(D.CLR, (rng.random(K) < 0.2).astype(float), pid=(np.arange(K) // 5).astype(np.int32))
    ds = api.Dataset(data)
    prior = api.create_prior("normal", variance=1.0)
    n = {}
    for r in (None, route):
        if r:
            monkeypatch.setenv("CYC_FIT_ROUTE", r)
        api.fit_cyclops_model(ds, prior)
        n0 = api.launch_count()
        fit = api.fit_cyclops_model(ds, prior)
        n[r] = (api.launch_count() - n0, fit)
    assert n[None][0] == n[route][0]
    np.testing.assert_array_equal(n[None][1].beta, n[route][1].beta)
