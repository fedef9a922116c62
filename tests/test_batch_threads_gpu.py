"""The 8-fit kernel at 256 and 512 threads a CTA and 1, 3 and 8 CTAs a group:
every fit of a CV grid, and of a batch under its own weights, is the oracle's
under the precision contract, cycle for cycle.  Columns of 5 to 20k entries
over 40k rows: batches of one column a warp that share rows, batches inside
and outside the batch cache, streamed and dense columns; 10 fits leave the
second group with 6 empty places."""
import numpy as np
import pytest

from conftest import assert_contract
from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


def _data(model, K=40_000, seed=3):
    rng = np.random.default_rng(seed)
    b = D.ColumnBuilder(K).intercept()
    eta = np.full(K, -1.0)
    pool = rng.choice(K, size=6_000, replace=False)
    for c in range(90):
        n = int(rng.integers(5, 600))
        rows = np.sort(rng.choice(pool, size=n, replace=False))
        vals = rng.normal(size=n)
        b.sparse(rows, vals)
        if c % 3 == 0:
            eta[rows] += 0.5 * vals
    x = rng.normal(size=K)
    b.dense(x)
    eta += 0.2 * x
    for n in np.maximum(20, 20_000 * np.arange(1, 151) ** -0.9).astype(int):
        b.indicator(np.sort(rng.choice(K, size=n, replace=False)))
    if model == D.LR:
        y = (rng.random(K) < 1.0 / (1.0 + np.exp(-eta))).astype(float)
    else:
        y = rng.poisson(np.exp(np.minimum(eta, 3.0))).astype(float)
    return b.build(model, y, has_intercept=True)


@pytest.mark.parametrize("model", [D.LR, D.PR])
@pytest.mark.parametrize("shape", ["1,256", "3,256", "8,256", "1,512", "3,512", "8,512"])
@pytest.mark.parametrize("weighted", [False, True])
def test_eight_fit_shapes_match_oracle(cuda_lib, monkeypatch, model, shape, weighted):
    from cyclops_b200 import api
    from oracle import oracle as O
    monkeypatch.setenv("CYC_BATCH_GROUP", "8")
    monkeypatch.setenv("CYC_BATCH_CLUSTER", shape)
    data = _data(model)
    tol = 1e-7
    ctl = api.create_control(tolerance=tol)
    prior = api.PriorSpec(D.PRIOR_LAPLACE, 1.0, [0])
    octl = O.make_control(tolerance=tol, convergence_type=D.CONV_GRADIENT)
    variances = [D.laplace_variance(lam) for lam in (1.0, 10.0)]
    masks = api.cv_fold_weights(data.K, 5, 31)
    if weighted:
        rng = np.random.default_rng(8)
        w = [m * rng.integers(0, 3, size=data.K) for m in masks] * 2
        fits = api.batch_fit(data, prior, np.repeat(variances, 5), weights=w, control=ctl)
    else:
        w = list(masks) * 2
        fits = api.cv_grid_fit(data, prior, api.fold_ids_from_weights(masks), 5, variances, ctl).fits
    assert api.last_run_stats()["cluster_ctas"] == int(shape.split(",")[0])
    for i in (0, 4, 7, 9):
        ref = O.port().fit(data, D.PRIOR_LAPLACE, variances[i // 5], control=octl, exclude=[0], weights=w[i])
        assert ref.return_flag == 0
        assert_contract(fits[i], ref, what=i)


@pytest.mark.parametrize("model", [D.LR, D.PR])
@pytest.mark.parametrize("shape", ["1,512", "3,512", "8,512"])
def test_eight_fit_shapes_mixed_precision(cuda_lib, monkeypatch, model, shape):
    """FP32 state with compensated sums, then the FP64 polish, both sides
    converged tightly (Mittal rule, 1e-12): the contract without cycle counts,
    as a change of 1e-12 is at the rounding of the likelihood's sum."""
    from cyclops_b200 import api
    from oracle import oracle as O
    monkeypatch.setenv("CYC_BATCH_GROUP", "8")
    monkeypatch.setenv("CYC_BATCH_CLUSTER", shape)
    data = _data(model, K=20_000, seed=7)
    masks = api.cv_fold_weights(data.K, 4, 13)
    variances = [D.laplace_variance(lam) for lam in (2.0, 20.0)]
    prior = api.PriorSpec(D.PRIOR_LAPLACE, 1.0, [0])
    ctl = api.create_control(tolerance=1e-12, convergence_type="mittal", precision="mixed", polish_tolerance=1e-5,
                             max_iterations=5000)
    res = api.cv_grid_fit(data, prior, api.fold_ids_from_weights(masks), 4, variances, ctl)
    octl = O.make_control(tolerance=1e-12, convergence_type=D.CONV_MITTAL, max_iterations=5000)
    for i in (0, 3, 6):
        ref = O.port().fit(data, D.PRIOR_LAPLACE, variances[i // 4], control=octl, exclude=[0], weights=masks[i % 4])
        assert_contract(res.fits[i], ref, iterations=False, what=i)
