"""The persistent loop of small matrices (jk_small.cu) against the general step kernels (taken when a
trace is asked for) and the oracle, bit for bit."""
import numpy as np
import pytest

import oracle
from jkogb_b200 import gen

pytestmark = pytest.mark.gpu


def _same(a, b):
    a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
    fa, fb = a.view(np.float64), b.view(np.float64)
    na, nb = np.isnan(fa), np.isnan(fb)
    return a.shape == b.shape and np.array_equal(na, nb) and np.array_equal(np.where(na, 0.0, fa).view(np.uint64),
                                                                            np.where(nb, 0.0, fb).view(np.uint64))


def _input(n, n_plus, cplx, form, seed):
    r = np.random.Generator(np.random.PCG64(seed))
    Y = r.standard_normal((n, n)) + (1j * r.standard_normal((n, n)) if cplx else 0.0)
    J = np.concatenate([np.ones(n_plus, np.int64), -np.ones(n - n_plus, np.int64)])
    if form == "graded":
        Y = Y * 10.0 ** r.uniform(-8, 0, n)[None, :]
        J = J[r.permutation(n)]
    if form == "tied":  # equal weights, zeros and zero columns
        Y = np.round(Y.real)
        Y[:, ::5] = 0.0
        J = J[r.permutation(n)]
        Y = Y + 0j if cplx else Y
    if form == "tiny":  # beside the straight-line forms' range
        Y = Y * 10.0 ** r.uniform(-160, 100, (n, n))
    return np.asfortranarray(Y), J


# cluster sizes 1 to 16, the largest orders, odd ones, all signs equal, N_2 below N/2
@pytest.mark.parametrize("n,n_plus,cplx,form,n_2,steps", [
    (3, 1, False, "gauss", 0, 0), (4, 4, False, "gauss", 0, 0), (5, 0, True, "gauss", 0, 0), (16, 12, False, "gauss", 3, 0),
    (17, 8, True, "gauss", 0, 0), (32, 16, False, "graded", 0, 0), (33, 17, False, "tied", 0, 0), (31, 20, True, "tied", 5, 0),
    (46, 23, False, "gauss", 0, 0), (64, 40, False, "graded", 0, 200), (70, 35, False, "tiny", 0, 40),
    (64, 32, True, "graded", 20, 60), (85, 30, True, "gauss", 0, 25), (97, 50, False, "gauss", 0, 120),
    (128, 64, False, "tied", 0, 60), (133, 66, False, "gauss", 0, 25), (24, 12, True, "tiny", 0, 40)])
def test_small_loop_equals_general_and_oracle(n, n_plus, cplx, form, n_2, steps):
    import jkogb_b200 as jk
    Y, J = _input(n, n_plus, cplx, form, 1000 + n)
    steps = steps or 20 * n + 50
    with np.errstate(all="ignore"):
        s = jk.step_loop(Y, J, n_2=n_2, max_steps=steps)
        g = jk.step_loop(Y, J, n_2=n_2, max_steps=steps, trace=True)
        o = oracle.step_loop(Y, J, n_2=n_2, nt=1, stop_after=steps)
    assert s["info"] == g["info"]
    for k in ("A", "U", "Z", "sigma"):
        assert _same(s[k], g[k]) and _same(s[k], o[k]), k


def test_small_loop_non_finite():
    """A non-finite entry ends the loop with the general kernels' INFO and results."""
    import jkogb_b200 as jk
    for cplx in (False, True):
        Y, J = _input(20, 11, cplx, "gauss", 7)
        Y[3, 12] = np.inf
        out = []
        for trace in (False, True):
            try:
                out.append(jk.step_loop(Y, J, trace=trace, max_steps=50)["info"])
            except jk.JkError as e:
                out.append(e.info)
        assert out[0] == out[1]
