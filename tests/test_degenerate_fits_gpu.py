"""Fits that cannot succeed end as the oracle's do: every weight zero, and an
overflowing predictor on a row without weight (0 * inf enters the sums, as in the
reference, whose engine multiplies every row's terms by its weight)."""
import numpy as np
import pytest

from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu

K = 900


def _data(model, overflow):
    rng = np.random.default_rng(model)
    b = D.ColumnBuilder(K).intercept()
    for n in (40, 200, 700):
        b.indicator(np.sort(rng.choice(np.arange(10, K), n, replace=False)))
    if overflow:
        b.indicator(np.arange(10))                     # the rows without weight
    y = (rng.random(K) < 0.4).astype(float) if model == D.LR else rng.poisson(1.0, K).astype(float)
    return b.build(model, y, has_intercept=True)


@pytest.mark.parametrize("route,shape", [("columns", "1,128,1"), ("cluster", "1,128,1"), ("cluster", "3,64,1"),
                                         ("cluster", "2,256,2")])
@pytest.mark.parametrize("kind", ["no weight", "overflow"])
@pytest.mark.parametrize("model", [D.LR, D.PR])
def test_ends_as_the_oracle(cuda_lib, monkeypatch, model, kind, route, shape):
    from cyclops_b200 import api
    from oracle import oracle as O
    monkeypatch.setenv("CYC_FIT_ROUTE", route)
    monkeypatch.setenv("CYC_BATCH_CLUSTER", shape)
    data = _data(model, kind == "overflow")
    w = np.zeros(K)
    start = None
    if kind == "overflow":
        w[10:] = 1.0
        start = np.zeros(data.J)
        start[-1] = 800.0
    want = O.port().fit(data, D.PRIOR_NORMAL, 1.0, weights=w, exclude=[0], start=start,
                        control=O.make_control(max_iterations=30))
    got = api.fit_cyclops_model(data, api.create_prior("normal", variance=1.0, exclude=[0]), weights=w,
                                control=api.create_control(max_iterations=30), starting_coefficients=start)
    assert got.return_flag == want.return_flag and got.iterations == want.iterations
    np.testing.assert_array_equal(np.isnan(got.beta), np.isnan(want.beta))
    np.testing.assert_allclose(got.beta, want.beta, rtol=1e-6, atol=1e-9)
    assert np.isnan(got.log_likelihood) == np.isnan(want.log_likelihood)
