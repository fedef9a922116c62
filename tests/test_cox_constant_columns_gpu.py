"""Cox columns that say nothing -- constant in every risk set, or of rows that
never share one with others -- have gradient and Hessian 0: a step of exactly 0
under a normal or Laplace prior, and no estimate (as the reference) under none."""
import numpy as np
import pytest

from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


def _data(K, strata, extra):
    rng = np.random.default_rng(K + strata)
    s = np.sort(rng.integers(0, max(1, strata), K)).astype(np.int32)
    t = rng.exponential(size=K)
    o = np.lexsort((-t, s))
    s, t = s[o], t[o]
    y = (rng.random(K) < 0.3).astype(float)
    b = D.ColumnBuilder(K)
    x = rng.normal(size=K)
    b.dense(x)
    if extra == "real":
        b.sparse(np.arange(K), np.full(K, 3.7))
    b.indicator(rng.choice(K, K // 3, replace=False))
    if extra == "rows":
        b.indicator(np.arange(K))
    elif extra == "stratum":
        b.indicator(np.flatnonzero(s == 1))
    j = {"rows": 2, "stratum": 2, "real": 1}[extra]
    return b.build(D.COX, y, pid=s, time=t), j


@pytest.mark.parametrize("shape", ["1,128", "4,128", "16,512"])
@pytest.mark.parametrize("K", [300, 20_000])
@pytest.mark.parametrize("strata,extra", [(0, "rows"), (7, "rows"), (7, "stratum"), (0, "real"), (7, "real")])
def test_columns_without_information(cuda_lib, monkeypatch, shape, K, strata, extra):
    from cyclops_b200 import api
    monkeypatch.setenv("CYC_COX_CLUSTER", shape)
    data, j = _data(K, strata, extra)
    ds = api.Dataset(data)
    for name in ("normal", "laplace"):
        fit = api.fit_cyclops_model(ds, api.create_prior(name, variance=1.0))
        assert fit.return_flag == 0 and fit.beta[j] == 0.0 and np.any(fit.beta != 0.0)
    flat = api.fit_cyclops_model(ds, api.create_prior("none"))
    assert np.isnan(flat.beta[j]) and flat.return_flag == 3
