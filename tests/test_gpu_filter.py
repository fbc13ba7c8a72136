"""The filtered exact ranking (jk_filter.cu) against the full column scan, which a loop with a trace
takes: A, U, Z, SIGMA and INFO bit for bit, where pairs are ambiguous and where they are not."""
import numpy as np
import pytest

from jkogb_b200 import gen

pytestmark = pytest.mark.gpu


def _bits(a):
    a = np.ascontiguousarray(a)
    f = a.view(np.float64)
    return np.where(np.isnan(f), 0.0, f).view(np.uint64), np.isnan(f)


def _input(n, n_plus, cplx, form):
    r = np.random.Generator(np.random.PCG64(n + 7))
    Y = r.standard_normal((n, n)) + (1j * r.standard_normal((n, n)) if cplx else 0.0)
    J = np.concatenate([np.ones(n_plus, np.int64), -np.ones(n - n_plus, np.int64)])
    if form != "sorted":
        J = J[r.permutation(n)]
    if form == "graded":
        Y = Y * 10.0 ** r.uniform(-9, 0, n)[None, :]
    elif form == "near":  # nearly diagonal: weights at the level of their rounding, over the filter's capacity
        Y = np.diag(r.uniform(0.5, 2.0, n)) + 1e-11 * 10.0 ** r.uniform(-8, 0, (n, n)) * Y
    elif form == "tiny":  # weights through the end of the exponent range, exact ties at zero
        Y = np.diag(r.uniform(0.5, 2.0, n)) + 10.0 ** r.uniform(-300, -100, (n, n)) * Y
    elif form == "tied":
        Y = np.round(Y.real) + (1j * np.round(Y.imag) if cplx else 0.0)
        Y[:, ::7] = Y[:, 1::7][:, :Y[:, ::7].shape[1]]
    elif form == "huge":  # squares beyond the numbers
        Y = Y * 1e160
    elif form == "small":
        Y = Y * 1e-170
    return np.asfortranarray(Y), J


@pytest.mark.parametrize("n,n_plus,cplx,form,n_2,steps", [
    (800, 400, False, "gauss", 0, 20), (901, 250, False, "graded", 0, 20), (1040, 520, False, "sorted", 0, 12),
    (800, 400, False, "near", 0, 80), (800, 400, False, "tiny", 0, 12), (801, 400, False, "tied", 0, 10),
    (800, 390, False, "huge", 0, 3), (800, 390, False, "small", 0, 4), (800, 400, False, "gauss", 100, 6),
    (110, 55, True, "gauss", 0, 40), (201, 60, True, "graded", 0, 30), (300, 150, True, "near", 0, 70),
    (364, 182, False, "gauss", 0, 20), (513, 256, False, "graded", 0, 30), (400, 200, False, "near", 0, 80),
    (401, 200, False, "tied", 0, 10), (86, 40, True, "graded", 0, 30),
    (1701, 850, False, "gauss", 0, 4), (1201, 600, True, "graded", 0, 3),  # the large Gram tiles, odd columns
    (203, 100, True, "tiny", 0, 12), (200, 100, True, "tied", 0, 10), (150, 70, True, "huge", 0, 3)])
def test_filter_equals_scan(n, n_plus, cplx, form, n_2, steps):
    import jkogb_b200 as jk
    Y, J = _input(n, n_plus, cplx, form)

    def go(trace):
        try:
            return jk.step_loop(Y, J, n_2=n_2, max_steps=steps, trace=trace)
        except jk.JkError as e:
            return dict(info=e.info)
    with np.errstate(all="ignore"):
        f, s = go(False), go(True)
    assert f["info"] == s["info"]
    for k in ("A", "U", "Z", "sigma"):
        if k in s:
            (a, na), (b, nb) = _bits(f[k]), _bits(s[k])
            assert np.array_equal(na, nb) and np.array_equal(a, b), k


def test_filter_whole_solve():
    """A whole complex solve, through the stretch where most pairs are ambiguous to the end."""
    import jkogb_b200 as jk
    Y, J = gen.complex_gaussian(120, seed=5)
    f, s = jk.step_loop(Y, J), jk.step_loop(Y, J, trace=True)
    assert f["info"] == s["info"] > 0
    for k in ("A", "U", "Z", "sigma"):
        assert np.array_equal(_bits(f[k])[0], _bits(s[k])[0]), k
