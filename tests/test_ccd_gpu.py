"""The one-fit persistent kernel (csrc/ccd.cu) against the FP64 oracle, at the
sizes where its parts meet: rounds of its threads over a column, CTAs without
entries or rows, one CTA and clusters; and batches run one fit to a cluster
against the same batches in 8-fit groups."""
import numpy as np
import pytest

from conftest import assert_contract
from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


def _edge_problem(model, K, seed):
    """Columns of 0, 1, 31..33, 127..129, 255..257, 511..513 and K - 1 entries
    (indicator and real-valued), beside an intercept and a dense column."""
    rng = np.random.default_rng(seed)
    sizes = [n for n in (0, 1, 31, 32, 33, 127, 128, 129, 255, 256, 257, 511, 512, 513, K - 1) if n < K]
    b = D.ColumnBuilder(K)
    grouped = model in (D.CLR, D.CPR)
    if not grouped:
        b.intercept().dense(rng.normal(size=K))
    eta = np.zeros(K)
    for n in sizes:                                   # sparse columns come before indicators
        rows = np.sort(rng.choice(K, size=n, replace=False))
        x = rng.normal(size=n)
        eta[rows] += 0.2 * x
        b.sparse(rows, x)
    for n in sizes:
        b.indicator(rng.choice(K, size=n, replace=False))
    pid = None
    if grouped:
        pid = np.sort(rng.integers(0, max(2, K // 6), size=K)).astype(np.int32)
        y = (rng.random(K) < 0.3).astype(float) if model == D.CLR else rng.poisson(0.5, size=K).astype(float)
    elif model == D.LR:
        y = (rng.random(K) < 1.0 / (1.0 + np.exp(1.0 - eta))).astype(float)
    else:
        y = rng.poisson(np.exp(np.clip(eta - 0.5, -5, 2))).astype(float)
    return b.build(model, y, pid=pid, has_intercept=not grouped)


def _oracle(data, prior, variance, weights=None, conv=D.CONV_GRADIENT, tol=1e-6, max_iter=1000, start=None):
    from oracle import oracle as O
    ctl = O.make_control(tolerance=tol, convergence_type=conv, max_iterations=max_iter)
    return O.port().fit(data, prior, variance, control=ctl, weights=weights, start=start)


@pytest.mark.parametrize("shape", ["1,64,1", "1,128,1", "1,256,2", "3,128,2", "8,256,2", "16,256,1"])
@pytest.mark.parametrize("model", [D.LR, D.PR, D.CLR, D.CPR])
@pytest.mark.parametrize("K", [40, 1100])
def test_edge_columns_match_oracle(cuda_lib, monkeypatch, shape, model, K):
    from cyclops_b200 import api
    monkeypatch.setenv("CYC_BATCH_CLUSTER", shape)
    data = _edge_problem(model, K, seed=K + model)
    w = np.random.default_rng(3).integers(0, 3, size=K).astype(float) if K > 40 else None
    for prior, name in ((D.PRIOR_LAPLACE, "laplace"), (D.PRIOR_NORMAL, "normal")):
        fit = api.fit_cyclops_model(data, api.create_prior(name, variance=0.5), weights=w)
        assert_contract(fit, _oracle(data, prior, 0.5, w), what=(shape, model, K, name))


@pytest.mark.parametrize("conv", [D.CONV_LANGE, D.CONV_MITTAL, D.CONV_ONE_STEP, D.CONV_ZHANG_OLES])
@pytest.mark.parametrize("shape", ["1,128,1", "4,256,2"])
def test_convergence_rules_match_oracle(cuda_lib, monkeypatch, shape, conv):
    from cyclops_b200 import api
    monkeypatch.setenv("CYC_BATCH_CLUSTER", shape)
    data = _edge_problem(D.LR, 700, seed=9)
    tol = 1e-4
    fit = api.fit_cyclops_model(data, api.create_prior("laplace", variance=0.5),
                                api.create_control(tolerance=tol, convergence_type=conv, max_iterations=500))
    assert_contract(fit, _oracle(data, D.PRIOR_LAPLACE, 0.5, conv=conv, tol=tol, max_iter=500), what=(shape, conv))


@pytest.mark.parametrize("rows_in_smem", ["1", "0"])
@pytest.mark.parametrize("model", [D.LR, D.PR])
@pytest.mark.parametrize("form", ["folds", "weights", "starts", "fixed", "swindle", "plain"])
def test_one_to_a_cluster_equals_eight_to_a_group(cuda_lib, monkeypatch, model, form, rows_in_smem):
    """Both run the same serial coordinate descent in FP64: they differ by
    the rounding of sums alone, far inside the contract."""
    from cyclops_b200 import api
    K, F = 1301, 9
    rng = np.random.default_rng(model + 1)
    data = _edge_problem(model, K, seed=31 + model)
    ds = api.Dataset(data)
    prior = api.create_prior("laplace", variance=0.3)
    fold = (rng.permutation(K) % 5).astype(np.int32)
    boot = [np.bincount(rng.integers(0, K, K), minlength=K).astype(float) if f % 3 else None for f in range(F)]
    starts = [rng.normal(0, 0.1, data.J) if f % 2 else None for f in range(F)]
    variances = np.exp(rng.uniform(-2, 1, F))
    monkeypatch.setenv("CYC_BATCH_XB_SMEM", rows_in_smem)

    def run(group):
        monkeypatch.setenv("CYC_BATCH_GROUP", group)
        if form == "folds":
            g = api.cv_grid_fit(ds, prior, fold, 5, variances[:2])
            return g.fits, g.pred_loglik
        kw = {"weights": dict(weights=boot), "starts": dict(starts=starts), "fixed": dict(fixed_coefficients=[3, 7]),
              "swindle": dict(control=api.create_control(use_kkt_swindle=True)), "plain": {}}[form]
        return api.batch_fit(ds, prior, variances, **kw), None

    one, pll1 = run("1")
    eight, pll8 = run("8")
    for f, (a, b) in enumerate(zip(one, eight)):
        assert_contract(a, b, what=(form, model, f))
    if pll1 is not None:
        np.testing.assert_allclose(pll1, pll8, rtol=1e-9)
