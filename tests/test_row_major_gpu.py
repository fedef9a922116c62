"""The row-major copy behind computeXBeta: linear predictors are the bits of
the column-by-column axpy (each product and each sum rounded), for every
column format, rows from one to more than the warps hold at a time, empty
rows and columns, and more columns than one batch of a warp."""
import numpy as np
import pytest

from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,J,dense", [(1, 1, 0), (37, 40, 2), (5_003, 33, 0), (5_003, 700, 3), (200_003, 9_000, 1),
                                       (1_300_001, 70, 1)])
def test_predictors_are_the_axpy_order(cuda_lib, K, J, dense):
    from cyclops_b200 import api
    rng = np.random.default_rng(K + J)
    b = D.ColumnBuilder(K).intercept()
    cols = [(np.arange(K), np.ones(K))]
    for j in range(J):
        n = int(rng.integers(0, min(K, 3 * max(1, K // max(J, 20))) + 1))
        rows = np.unique(rng.integers(0, max(1, K - K // 10), size=n))      # the last tenth: dense columns only
        if j % 3 == 1:
            x = rng.normal(size=rows.size)
            b.sparse(rows, x)
        else:
            x = np.ones(rows.size)
            b.indicator(rows)
        cols.append((rows, x))
        if j < dense:
            x = rng.normal(size=K)
            b.dense(x)
            cols.append((np.arange(K), x))
    data = b.build(D.PR, (rng.random(K) < 0.3).astype(float), has_intercept=True)
    beta = rng.normal(size=data.J) * (rng.random(data.J) < 0.8)
    beta[0] = 0.5
    want = np.zeros(K)
    for j, (rows, x) in enumerate(cols):
        if beta[j] != 0.0:
            want[rows] = want[rows] + beta[j] * x
    eng = api.Engine(api.Dataset(data))
    eng.compute_xbeta(beta)
    np.testing.assert_array_equal(eng.get_xbeta(), want)
