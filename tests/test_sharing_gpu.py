"""Fits that share the device with others take clusters that run side by side,
and give the fits they give alone."""
import pytest

from conftest import assert_contract
from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", ["lr", "clr"])
def test_shared_fits_are_smaller_and_the_same(cuda_lib, model):
    from cyclops_b200 import api
    data = (D.synth_logistic(K=300_000, P=120, density=0.004, n_true=20, seed=5, zipf=1.1) if model == "lr" else
            D.synth_conditional(K=300_000, P=60, density=0.03))
    ds = api.Dataset(data)
    prior = api.create_prior("laplace", variance=1.0, exclude=[0] if model == "lr" else None)
    alone = api.batch_fit(ds, prior, [1.0])[0]
    ctas = api.last_run_stats()["cluster_ctas"]
    single = api.fit_cyclops_model(ds, prior)
    ds.share(16)
    shared = api.batch_fit(ds, prior, [1.0])[0]
    assert api.last_run_stats()["cluster_ctas"] < ctas and 16 * api.last_run_stats()["cluster_ctas"] <= 148
    assert_contract(shared, alone)
    assert_contract(api.fit_cyclops_model(ds, prior), single)
    ds.share(1)
    again = api.batch_fit(ds, prior, [1.0])[0]
    assert api.last_run_stats()["cluster_ctas"] == ctas and (again.beta == alone.beta).all()


def test_at_least_one_call(cuda_lib):
    from cyclops_b200 import _native, api
    ds = api.Dataset(D.synth_logistic(K=100, P=5, density=0.2, n_true=2, seed=1))
    with pytest.raises(_native.CyclopsError):
        ds.share(0)
