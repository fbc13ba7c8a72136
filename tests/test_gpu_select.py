"""The partner ranking and the greedy matching against the oracle's selection, at the orders where
the keys per thread, the threads or the blocks change, over weights that the short keys separate,
share in small groups, share in groups too long for them, and spread over the whole exponent range."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _weights(form, n, P, Q, rng):
    m = len(P)
    if form == "spread":      # both signs, most lists without a shared short key
        return rng.standard_normal(m) * np.exp(rng.uniform(-30, 10, m))
    if form == "groups":      # a few partners of every list differ in their last bits only
        base = rng.uniform(-1, 4, 4 * n)[rng.integers(0, 4 * n, m)]
        return (base.view(np.int64) + rng.integers(0, 3, m)).view(np.float64)
    if form == "long":        # groups beyond the short keys' limit, and many that are all equal
        base = np.array([1.0, -2.0, 0.0, -0.0, 7.0])[rng.integers(0, 5, m)]
        return np.where(base == 7.0, (base.view(np.int64) + rng.integers(0, 4, m)).view(np.float64), base)
    if form == "range":       # through zero, the denormal numbers and infinity
        w = np.ldexp(rng.choice([-1.0, 1.0], m), rng.integers(-1074, 1024, m))
        w[rng.uniform(size=m) < 0.05] = 0.0
        w[rng.uniform(size=m) < 0.01] = np.inf
        w[rng.uniform(size=m) < 0.2] = np.nan
        return w
    # every list prefers the same vertices, so that the lists are walked far
    c = np.exp(rng.uniform(-20, 0, n))
    return c[P - 1] + c[Q - 1] * (1.0 + 1e-9 * rng.standard_normal(m))


@pytest.mark.parametrize("n", [2, 65, 256, 257, 301, 512, 513, 601, 901, 1025, 2049])
@pytest.mark.parametrize("form", ["spread", "groups", "long", "range", "star"])
def test_selection(n, form):
    import jkogb_b200 as jk
    rng = np.random.Generator(np.random.PCG64(n))
    P, Q, _ = oracle.pairs(n, np.ones(n, np.int32), 1)
    w = _weights(form, n, P, Q, rng)
    W = np.full((n, n), np.nan)
    W[P - 1, Q - 1] = w
    W[Q - 1, P - 1] = w
    for n2 in {max(n // 3, 1), n // 2}:
        assert np.array_equal(jk.select(W, n2), oracle.select(n, w, P, Q, n2, id_ncp=2, nt=8)), n2
