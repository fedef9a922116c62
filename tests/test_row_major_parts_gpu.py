"""The row-major copy of designs with more columns than one part of its splits
holds (7,081): the bits of the column-by-column axpy."""
import numpy as np
import pytest

from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,J", [(701, 7_080), (701, 7_081), (701, 22_000)])
def test_predictors_are_the_axpy_order(cuda_lib, K, J):
    from cyclops_b200 import api
    rng = np.random.default_rng(J)
    b = D.ColumnBuilder(K).intercept()
    cols = [(np.arange(K), np.ones(K))]
    for j in range(J):
        rows = np.unique(rng.integers(0, K, size=int(rng.integers(0, 6))))
        x = rng.normal(size=rows.size) if j % 3 == 1 else np.ones(rows.size)
        if j % 3 == 1:
            b.sparse(rows, x)
        else:
            b.indicator(rows)
        cols.append((rows, x))
        if j % 9_000 == 8_500:
            x = rng.normal(size=K)
            b.dense(x)
            cols.append((np.arange(K), x))
    data = b.build(D.PR, (rng.random(K) < 0.3).astype(float), has_intercept=True)
    beta = rng.normal(size=data.J)
    want = np.zeros(K)
    for j, (rows, x) in enumerate(cols):
        want[rows] = want[rows] + beta[j] * x
    eng = api.Engine(api.Dataset(data))
    eng.compute_xbeta(beta)
    np.testing.assert_array_equal(eng.get_xbeta(), want)
