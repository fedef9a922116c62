"""The engine's calls that end in a kernel's own signal to the host: gradient,
update, objective and log likelihood of columns that take one block and
several, on engines that follow one another (and so share pinned blocks),
against NumPy in 64 bits.

Tolerance: sums of at most 5,000 terms of either sign, each within a few
ulps of its exact value: 5,000 * 2^-53 * 4 = 2.2e-12 of the sum of absolute
values; 1e-11 of that is asserted."""
import numpy as np
import pytest

from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 1024, 1025, 5000])
def test_signalled_calls_match_numpy(cuda_lib, n):
    from cyclops_b200 import api
    K = 6000
    rng = np.random.default_rng(n)
    rows = np.sort(rng.choice(K, size=n, replace=False))
    x = rng.normal(size=n)
    y = (rng.random(K) < 0.4).astype(float)
    data = D.ColumnBuilder(K).intercept().sparse(rows, x).indicator(rows).build(D.LR, y, has_intercept=True)
    ds = api.Dataset(data)
    for _ in range(2):
        eng = api.Engine(ds)
        eng.set_weights(None)
        eng.compute_fixed_terms_in_gradient_and_hessian()
        xb = np.full(K, 0.25)
        eng.compute_xbeta(np.array([0.25, 0.0, 0.0]))
        eng.compute_remaining_statistics()
        for j, xj, delta in ((1, x, -0.5), (2, np.ones(n), 0.125), (1, x, 0.75)):
            p = 1.0 / (1.0 + np.exp(-xb[rows]))
            g, h = eng.compute_gradient_and_hessian(j)
            assert abs(g - ((p - y[rows]) * xj).sum()) <= 1e-11 * np.abs(xj).sum()
            assert abs(h - (p * (1 - p) * xj * xj).sum()) <= 1e-11 * (xj * xj).sum()
            eng.update_xbeta(delta, j)
            xb[rows] = xb[rows] + delta * xj
        assert np.max(np.abs(eng.get_xbeta() - xb)) <= 1e-11
        assert abs(eng.get_gradient_objective() - (xb * y).sum()) <= 1e-11 * np.abs(xb).sum()
        want = (y * xb - np.log1p(np.exp(xb))).sum()
        assert abs(eng.get_log_likelihood() - want) <= 1e-11 * (np.abs(xb) + 1.0).sum()
        eng.update_xbeta(0.0, 1)                       # nothing to do
        assert np.array_equal(eng.get_xbeta(), eng.get_xbeta())
        del eng
