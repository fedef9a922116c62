"""Runs of short columns that share no row, a warp a column, against the FP64
oracle and against the kernel without runs: columns of 0 to 256 entries around the
warps' rounds, runs that a shared row, a long or dense column or the staging of
128 columns ends, weights, folds, held columns and starting values."""
import numpy as np
import pytest

from conftest import assert_contract
from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


def _data(model, K=9000, J=300, offset=False, seed=0):
    rng = np.random.default_rng(seed + model)
    b = D.ColumnBuilder(K)
    if offset:
        b.dense(rng.normal(size=K) * 0.1)
    b.intercept()
    sizes = [0, 1, 3, 31, 32, 33, 64, 96, 97, 255, 256, 257, 700]
    for j in range(J):
        n = sizes[j % len(sizes)] if j % 3 == 0 else int(rng.integers(1, 9))
        if j % 11 == 5:                                  # beside the column before it, on one of its rows
            rows = np.unique(np.append(rng.choice(K, n, replace=False), rows[:1]))
        else:
            rows = np.sort(rng.choice(K, n, replace=False))
        if j < J // 3:
            b.sparse(rows, rng.normal(size=rows.size))
        else:
            b.indicator(rows)
        if j in (50, 51):
            b.dense(rng.normal(size=K))
    y = (rng.random(K) < 0.4).astype(float) if model == D.LR else rng.poisson(0.8, K).astype(float)
    return b.build(model, y, has_intercept=True, has_offset=offset)


@pytest.mark.parametrize("in_smem", ["1", "0"])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("model", [D.LR, D.PR])
def test_runs_match_oracle(cuda_lib, monkeypatch, model, weighted, in_smem):
    from cyclops_b200 import api
    from oracle import oracle as O
    monkeypatch.setenv("CYC_BATCH_CLUSTER", "1,256,0")
    monkeypatch.setenv("CYC_BATCH_XB_SMEM", in_smem)
    data = _data(model)
    w = np.random.default_rng(1).integers(0, 3, data.K).astype(float) if weighted else None
    for prior, name in ((D.PRIOR_LAPLACE, "laplace"), (D.PRIOR_NORMAL, "normal")):
        want = [O.port().fit(data, prior, v, weights=w, exclude=[0]) for v in (0.5, 0.02)]
        got = api.batch_fit(data, api.create_prior(name, exclude=[0]), [0.5, 0.02], [w, w])
        for a, b in zip(got, want):
            assert_contract(a, b, what=(model, name, weighted, in_smem))


@pytest.mark.parametrize("form", ["folds", "held", "starts", "offset", "lange", "swindle", "mixed"])
def test_runs_equal_no_runs(cuda_lib, monkeypatch, form):
    from cyclops_b200 import api
    data = _data(D.PR, offset=form == "offset", seed=7)
    ds = api.Dataset(data)
    prior = api.create_prior("laplace", 0.3, exclude=[1 if form == "offset" else 0])
    ctl = {"lange": api.create_control(convergence_type="lange"), "swindle": api.create_control(use_kkt_swindle=True),
           "mixed": api.create_control(precision="mixed")}.get(form, api.create_control())
    start = np.random.default_rng(5).normal(0, 0.1, data.J)
    fold = (np.random.default_rng(6).permutation(data.K) % 3).astype(np.int32)

    def run():
        if form == "folds":
            g = api.cv_grid_fit(ds, prior, fold, 3, [0.3], ctl)
            return g.fits, g.pred_loglik
        kw = {"held": dict(fixed_coefficients=[3, 40, 41, 200]), "starts": dict(starts=[start, None])}.get(form, {})
        return api.batch_fit(ds, prior, [0.3, 0.05], control=ctl, **kw), None
    monkeypatch.setenv("CYC_BATCH_CLUSTER", "1,256,0")
    a, pa = run()
    monkeypatch.setenv("CYC_BATCH_CLUSTER", "1,256,1")
    b, pb = run()
    for x, y in zip(a, b):
        assert_contract(x, y, what=form, iterations=form != "mixed")
    if pa is not None:
        np.testing.assert_allclose(pa, pb, rtol=1e-9)


def test_plan_and_rule(cuda_lib):
    """Very short columns take runs by themselves: the same fits, one launch."""
    from cyclops_b200 import api
    d = D.synth_logistic(K=4000, P=3000, density=0.0012, n_true=20, seed=3)
    ds = api.Dataset(d)
    prior = api.create_prior("laplace", 1.0, exclude=[0])
    one = api.batch_fit(ds, prior, [1.0])[0]
    assert api.last_run_stats()["cluster_ctas"] == 1
    assert_contract(one, api.fit_cyclops_model(ds, api.create_prior("laplace", 1.0, exclude=[0])))
