"""The 2x2 HSVD's straight-line form and its hand-over to the general one: blocks at every scale, with
off-diagonals down through the exponent range (cosines that round to 1 or just below it), bit for bit
against the oracle."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _bits(a):
    f = np.ascontiguousarray(a).view(np.float64)
    return np.where(np.isnan(f), 0.0, f).view(np.uint64), np.isnan(f)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("J", [(1, 1), (1, -1), (-1, 1)])
def test_scales(cplx, J):
    import jkogb_b200 as jk
    rng = np.random.Generator(np.random.PCG64(5 + cplx))

    def draw():
        x = rng.standard_normal((2, 2))
        return x + 1j * rng.standard_normal((2, 2)) if cplx else x
    B = []
    for scale in (-1074, -1022, -1000, -700, -601, -600, -599, -300, 0, 300, 599, 600, 601, 700, 1000, 1020):
        for off in (0, 1, 5, 25, 26, 27, 28, 52, 53, 54, 60, 200, 599, 600, 601, 1000, 1075):
            b = draw()
            m = np.array([[0, -off], [-off, rng.integers(-3, 1)]])
            # (the parts by themselves: a complex product would make NaN of 0 times infinity)
            part = lambda v: np.ldexp(np.ldexp(v, m), scale)
            B.append(part(b.real) + 1j * part(b.imag) if cplx else part(b))
    B = np.array(B)
    Js = np.tile(np.array(J, np.int32), (len(B), 1))
    A, U, Z, info = jk.hsvd2_batch(B, Js, 1.0)
    for k in range(len(B)):
        a, u, z, inf = oracle.hsvd2(B[k], Js[k], 1.0)
        assert inf == info[k], k
        if inf < 0:
            continue
        for x, y in ((A[k], a), (U[k], u), (Z[k], z)):
            (p, pn), (q, qn) = _bits(x), _bits(np.asarray(y, x.dtype))
            assert np.array_equal(pn, qn) and np.array_equal(p, q), k
