"""Conditional models at linear predictors far from zero.  The conditional
likelihood does not see a shift common to a stratum, so a covariate such as a
calendar year reaches exp(500) with ordinary ratios; the solver must not form a
square of such a sum that no denominator has divided."""
import numpy as np
import pytest

from conftest import assert_contract
from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


def _problem(model, shift, strata=120, per=5):
    rng = np.random.default_rng(7)
    K = strata * per
    z = rng.normal(size=K)
    b = D.ColumnBuilder(K).dense(shift + z).sparse(np.arange(K), rng.normal(size=K))
    b.indicator(rng.choice(K, K // 3, replace=False))
    e = 0.6 * z
    if model == D.CLR:
        y = np.zeros(K)
        for s in range(strata):
            p = np.exp(e[per * s:per * s + per])
            y[per * s + rng.choice(per, p=p / p.sum())] = 1.0
    else:
        y = rng.poisson(0.7 * np.exp(e)).astype(float)
    return b.build(model, y, pid=np.repeat(np.arange(strata), per).astype(np.int32))


@pytest.mark.parametrize("shape", ["1,128,1", "1,256,1", "3,64,1"])
@pytest.mark.parametrize("shift", [0.0, 1000.0])
@pytest.mark.parametrize("model", [D.CLR, D.CPR])
@pytest.mark.parametrize("prior,name", [(D.PRIOR_LAPLACE, "laplace"), (D.PRIOR_NORMAL, "normal")])
def test_shared_shift_matches_oracle(cuda_lib, monkeypatch, shape, shift, model, prior, name):
    from cyclops_b200 import api
    from oracle import oracle as O
    monkeypatch.setenv("CYC_BATCH_CLUSTER", shape)
    data = _problem(model, shift)
    want = O.port().fit(data, prior, 10.0)
    assert want.return_flag == 0 and np.abs(data.column(0)[1] * want.beta[0]).max() > (370.0 if shift else 0.5)
    assert_contract(api.fit_cyclops_model(data, api.create_prior(name, variance=10.0)), want, what=(shape, shift))
    assert_contract(api.batch_fit(data, api.create_prior(name), [10.0])[0], want, what=("batch", shape, shift))
