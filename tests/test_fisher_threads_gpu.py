"""Fisher information of datasets of different row counts from several host
threads at once: each call's shared-memory bitmap has its own size, and no call
may take another's launch limit away."""
import threading

import numpy as np
import pytest

from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


def _dataset(K, seed):
    rng = np.random.default_rng(seed)
    b = D.ColumnBuilder(K)
    for n in (200, 100, 50):
        b.indicator(rng.choice(K, n, replace=False))
    return b.build(D.LR, (rng.random(K) < 0.3).astype(float))


def test_calls_of_different_sizes_do_not_disturb_each_other(cuda_lib):
    from cyclops_b200 import api
    sets = [api.Dataset(_dataset(K, K)) for K in (1_500_000, 400_000, 1_200_000, 600_000) * 2]
    engines = []
    for ds in sets:
        e = api.Engine(ds)
        e.set_weights(None)
        e.compute_xbeta(np.zeros(3))
        e.compute_remaining_statistics()
        engines.append(e)
    cols = [0, 1, 2]
    want = [e.fisher_information(cols) for e in engines]
    for w in want:
        np.testing.assert_allclose(np.diag(w), np.array([200, 100, 50]) * 0.25, rtol=1e-12)
    failed = []

    def work(e, w):
        try:
            for _ in range(1500):
                np.testing.assert_array_equal(e.fisher_information(cols), w)
        except Exception as x:                                  # noqa: BLE001
            failed.append(x)
    threads = [threading.Thread(target=work, args=a) for a in zip(engines, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed
