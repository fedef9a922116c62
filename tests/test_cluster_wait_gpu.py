"""The bounded waits between the CTAs of a fit: where one CTA is lost (its wait
given up on the host's word, CYC_WAIT_CLOCKS), the cluster stops together, the
call returns the timeout status, and the device goes on to serve the same fit.
Others wait 20 million clocks, about ten milliseconds."""
import numpy as np
import pytest

from conftest import assert_contract
from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


def _data(model, K=1500):
    rng = np.random.default_rng(model)
    b = D.ColumnBuilder(K)
    if model in (D.LR, D.PR):
        b.intercept()
    b.sparse(np.arange(K), rng.normal(size=K))
    for n in (40, 400, K // 2):
        b.indicator(rng.choice(K, n, replace=False))
    y = (rng.random(K) < 0.3).astype(float)
    pid = np.sort(rng.integers(0, K // 5, K)).astype(np.int32) if model in (D.CLR, D.CPR) else \
        np.zeros(K, np.int32) if model == D.COX else None
    time = np.arange(K, 0, -1, dtype=float) if model == D.COX else None
    return b.build(model, y, pid=pid, time=time, has_intercept=model in (D.LR, D.PR))


@pytest.mark.parametrize("conv", [D.CONV_GRADIENT, D.CONV_ONE_STEP])
@pytest.mark.parametrize("limit", ["20000000,0", "20000000,2", "0"])
@pytest.mark.parametrize("model,shape", [(D.LR, "4,128,1"), (D.PR, "4,256,2"), (D.CLR, "3,128,1"), (D.COX, "4,128"),
                                         (D.COX, "16,512")])
def test_lost_cta_is_a_timeout(cuda_lib, monkeypatch, model, shape, limit, conv):
    from cyclops_b200 import _native, api
    monkeypatch.setenv("CYC_BATCH_CLUSTER" if model != D.COX else "CYC_COX_CLUSTER", shape)
    data = _data(model)
    ds = api.Dataset(data)
    prior = api.create_prior("laplace", variance=1.0)
    ctl = api.create_control(convergence_type=conv, max_iterations=50)
    want = api.fit_cyclops_model(ds, prior, ctl)
    monkeypatch.setenv("CYC_WAIT_CLOCKS", limit)
    with pytest.raises(_native.CyclopsError) as e:
        api.fit_cyclops_model(ds, prior, ctl)
    assert "ran out" in str(e.value)
    if conv == D.CONV_GRADIENT:
        with pytest.raises(_native.CyclopsError):
            api.batch_fit(ds, prior, [1.0, 0.5], control=ctl)
    monkeypatch.delenv("CYC_WAIT_CLOCKS")
    again = api.fit_cyclops_model(ds, prior, ctl)
    np.testing.assert_array_equal(again.beta, want.beta)
    assert_contract(again, want)
