"""Fisher information of every pair of columns against NumPy in 64 bits: each
column format on either side of a pair, columns on both sides of the block /
warp split (2,048 entries), an empty column and a repeated one, and rows that
fit the bitmap of a block and rows that do not (1.6M).

Tolerance: a thread adds at most K / 256 terms in sequence, a warp 2,048 / 32,
and the terms of a pair add up in absolute value to at most the geometric
mean of the two columns' own sums (Cauchy-Schwarz); a term carries under 8
roundings.  (K / 256 + 24) * 2^-53 of that mean is at most 7.4e-13 for 1.7M
rows, and the grouped models subtract a second such sum: 2e-12."""
import numpy as np
import pytest

from cyclops_b200 import data as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model,K", [("lr", 7_003), ("pr", 7_003), ("clr", 7_003), ("lr", 1_700_001)])
def test_pairs_match_numpy(cuda_lib, model, K):
    from cyclops_b200 import api
    m = {"lr": D.LR, "pr": D.PR, "clr": D.CLR}[model]
    rng = np.random.default_rng(K + m)
    b = D.ColumnBuilder(K)
    X = []
    if model != "clr":
        b.intercept()
        X.append((np.arange(K), np.ones(K)))
    x = rng.normal(size=K)
    b.dense(x)
    X.append((np.arange(K), x))
    for n in (2048, 1, 2049, 33, 0, 3000, 257):
        rows = np.sort(rng.choice(K, size=n, replace=False)).astype(np.int64)
        b.indicator(rows)
        X.append((rows, np.ones(n)))
        rows = np.sort(rng.choice(K, size=n, replace=False)).astype(np.int64)
        x = rng.normal(size=n)
        b.sparse(rows, x)
        X.append((rows, x))
    pid = None
    y = (rng.random(K) < 0.3).astype(float)
    if model == "clr":
        pid = np.sort(rng.integers(0, K // 5, size=K)).astype(np.int32)
        data = b.build(m, y, pid=pid)
    else:
        data = b.build(m, y, has_intercept=True)
    beta = rng.normal(0.0, 0.2, size=data.J)
    eng = api.Engine(api.Dataset(data))
    eng.compute_xbeta(beta)
    eng.compute_remaining_statistics()
    cols = list(range(data.J)) + [1]
    got = eng.fisher_information(cols)
    xb = eng.get_xbeta()
    e = np.exp(xb)
    if model == "lr":
        v = e / (1 + e) - (e / (1 + e)) ** 2
    elif model == "pr":
        v = e
    else:
        s = np.concatenate([[0], np.cumsum(pid[1:] != pid[:-1])])
        den = np.bincount(s, e)
        v = e / den[s]
    dense = np.zeros(K)
    want = np.zeros((len(cols), len(cols)))
    info = np.zeros(len(cols))
    t = [np.bincount(s[X[c][0]], e[X[c][0]] * X[c][1], len(den)) for c in cols] if model == "clr" else None
    for i, ci in enumerate(cols):
        dense[:] = 0.0
        dense[X[ci][0]] = X[ci][1]
        for j, cj in enumerate(cols):
            rows, xj = X[cj]
            want[i, j] = (v[rows] * dense[rows] * xj).sum()
            if i == j:
                info[i] = want[i, i]
            if model == "clr":
                want[i, j] -= (t[i] * t[j] / den ** 2).sum()
    scale = np.sqrt(np.outer(info, info))
    assert np.all(np.abs(got - want) <= 2e-12 * scale)
    np.testing.assert_array_equal(got, got.T)
