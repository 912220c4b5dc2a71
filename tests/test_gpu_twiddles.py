"""The twiddle tables that the transforms fill: cosines and sines to two units of 2^-53 of long double ones, the
eight-fold symmetry bit for bit, the same bits for the same angle at every length, and the inverse's table the
conjugate of the forward one."""
import numpy as np
import pytest

import qmctoolscl_gb300 as q

pytestmark = pytest.mark.gpu
U = np.uint64
PI = np.longdouble("3.14159265358979323846264338327950288")


def _tables(m):
    n = 1 << m
    out = []
    for f in (q.fft_bro_1d_radix2, q.ifft_bro_1d_radix2):
        t = np.full(n, np.nan), np.full(n, np.nan)
        f(U(1), U(1), U(n // 2), *t, np.zeros(n), np.zeros(n))
        out.append(t)
    return out


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 9, 12, 17])
def test_twiddles(m):
    n = 1 << m
    (c, s), (ci, si) = _tables(m)
    a = 2 * PI * np.arange(n, dtype=np.longdouble) / n
    assert np.abs(c - np.cos(a)).max() <= 2.0 ** -52 and np.abs(s + np.sin(a)).max() <= 2.0 ** -52
    assert np.array_equal(ci, c) and np.array_equal(si, -s)
    t = np.arange(n)
    assert np.array_equal(c[-t % n], c) and np.array_equal(s[-t % n], -s)
    if n >= 4:
        quarter = (t + n // 4) % n
        assert np.array_equal(c[quarter], s) and np.array_equal(s[quarter], -c)
    if m > 1:
        (h, k), _ = _tables(m - 1)
        assert np.array_equal(c[::2], h) and np.array_equal(s[::2], k)
