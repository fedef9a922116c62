"""Cox batches whose risk sets do not fit the device together run in parts: the
same fits and scores, a launch a part."""
import numpy as np
import pytest

from conftest import assert_contract
from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


def _data(K=1500):
    rng = np.random.default_rng(1)
    b = D.ColumnBuilder(K)
    b.sparse(np.arange(K), rng.normal(size=K))
    for n in (60, 300, 700):
        b.indicator(rng.choice(K, n, replace=False))
    return b.build(D.COX, (rng.random(K) < 0.3).astype(float), pid=np.zeros(K, np.int32),
                   time=np.arange(K, 0, -1, dtype=float))


@pytest.mark.parametrize("bound,parts", [("1", 7), ("400000", None)])
def test_replicates_in_parts(cuda_lib, monkeypatch, bound, parts):
    from cyclops_b200 import api
    ds = api.Dataset(_data())
    rng = np.random.default_rng(3)
    K, F = 1500, 7
    weights = [np.bincount(rng.integers(0, K, K), minlength=K).astype(float) if f else None for f in range(F)]
    prior = api.create_prior("laplace", variance=0.5)
    whole = api.batch_fit(ds, prior, [0.5] * F, weights)
    assert api.last_run_stats()["launches"] == 1
    cycles = api.last_run_stats()["cycles"]
    monkeypatch.setenv("CYC_COX_BATCH_BYTES", bound)
    cut = api.batch_fit(ds, prior, [0.5] * F, weights)
    n = api.last_run_stats()["launches"]
    assert n == parts if parts else 1 < n < F
    assert api.last_run_stats()["cycles"] == cycles
    for f, (a, b) in enumerate(zip(cut, whole)):
        assert_contract(a, b, what=f)


def test_cross_validation_in_parts(cuda_lib, monkeypatch):
    from cyclops_b200 import api
    ds = api.Dataset(_data())
    fold = (np.random.default_rng(4).permutation(1500) % 5).astype(np.int32)
    prior = api.create_prior("laplace", variance=0.5)
    whole = api.cv_grid_fit(ds, prior, fold, 5, [0.1, 1.0])
    monkeypatch.setenv("CYC_COX_BATCH_BYTES", "1")
    cut = api.cv_grid_fit(ds, prior, fold, 5, [0.1, 1.0])
    for f, (a, b) in enumerate(zip(cut.fits, whole.fits)):
        assert_contract(a, b, what=f)
    np.testing.assert_allclose(cut.pred_loglik, whole.pred_loglik, rtol=1e-9)
