"""An update by zero, and an update of a column without entries, leave the
engine's state as it was: linear predictors, statistics, objective."""
import numpy as np
import pytest

from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [D.LR, D.PR, D.CLR, D.CPR, D.COX])
def test_updates_that_move_nothing(cuda_lib, model):
    from cyclops_b200 import api
    K = 3000
    rng = np.random.default_rng(model)
    b = D.ColumnBuilder(K).sparse(np.arange(0, K, 2), rng.normal(size=K // 2)).sparse(np.zeros(0, int), np.zeros(0))
    b.indicator(rng.choice(K, 900, replace=False))
    pid = {D.CLR: np.arange(K) // 6, D.CPR: np.arange(K) // 6, D.COX: np.zeros(K)}.get(model)
    data = b.build(model, (rng.random(K) < 0.4).astype(float), pid=None if pid is None else pid.astype(np.int32),
                   time=np.arange(K, 0, -1, dtype=float) if model == D.COX else None)
    eng = api.Engine(api.Dataset(data))
    eng.set_weights(None)
    eng.compute_fixed_terms_in_gradient_and_hessian()
    eng.compute_xbeta(np.array([0.3, 2.0, -0.2]))
    eng.compute_remaining_statistics()

    def state():
        eng.compute_numerator_for_gradient(0)
        return (eng.get_xbeta(), np.array(eng.compute_gradient_and_hessian(0)), eng.get_log_likelihood(),
                eng.get_gradient_objective())
    before = state()
    assert np.any(before[0] != 0.0)
    eng.update_xbeta(0.0, 0)
    eng.update_xbeta(0.5, 1)                            # no entries
    for x, y in zip(before, state()):
        np.testing.assert_array_equal(x, y)
    eng.update_xbeta(0.25, 0)
    assert np.any(eng.get_xbeta() != before[0])
