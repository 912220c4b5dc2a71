"""The FP64 fused transforms with scales and data near the ends of a double's range: lam constant, so that
the exact result is the data times scale * lam (or / lam).  Tolerance: 2e-15 of the vector's norm (numpy's and
the FP64 stages' own errors are 2 to 4e-16), and below the normal range half a unit (2^-1075) per rounding, at most
16 n of them in an output.  What is out of range above is not finite.  The complex quotient takes |lam|^2, which has
to be a double: lam = 2^+-600 is left to the real form there."""
import numpy as np
import pytest

from qmctoolscl_gb300 import tc_fft

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,nv", [(9, 200), (10, 2), (13, 2), (17, 1)])
@pytest.mark.parametrize("divide", [False, True])
@pytest.mark.parametrize("log2_scale,magnitude,log2_lam", [
    (-800, 1e-70, 0), (800, 1e80, 0), (-800, 1e70, 0), (800, 1e-80, 0), (-100, 1e-200, 0), (120, 1e200, 0), (-75, 1e-250, 0),
    (0, 1e298, 18), (0, 1e-300, -18), (300, 1e200, -300), (-300, 1e-200, 300), (0, 1.0, 600), (0, 1.0, -600)])
def test_scales(m, nv, divide, log2_scale, magnitude, log2_lam):
    rng = np.random.Generator(np.random.SFC64(m))
    n = 1 << m
    z = rng.standard_normal((nv, n)) * magnitude
    scale, lam = 2.0 ** log2_scale, np.full(n, 2.0 ** (-log2_lam if divide else log2_lam))
    want = (z.astype(np.longdouble) * np.ldexp(np.longdouble(1), log2_scale + log2_lam))
    x, xr, xi = z.copy(), z.copy(), np.zeros_like(z)
    tc_fft.fwht_mul_fwht(nv, 1, n // 2, lam, x, divide=divide, scale=scale)
    if not divide or abs(log2_lam) < 512:
        tc_fft.fft_mul_ifft(nv, 1, n // 2, lam, np.zeros(n), xr, xi, divide=divide, scale=scale)
    else:
        xr = x
    top = np.abs(want).max()
    if top > 1e308:
        assert not np.isfinite(x).any() and not np.isfinite(xr).any()
        return
    low = 16 * n * 2.0 ** -1074
    for y in (x, xr):
        assert np.isfinite(y).all()
        err = np.sqrt((((y - want) / top) ** 2).sum(axis=1)) / np.sqrt(((want / top) ** 2).sum(axis=1))
        assert (np.abs(y - want) <= low).all() or err.max() < 2e-15, err.max()
    assert np.abs(xi).max() <= max(low, 1e-13 * float(top))


@pytest.mark.parametrize("m,nv", [(9, 200), (10, 2), (12, 2), (13, 2), (17, 1), (20, 1)])
@pytest.mark.parametrize("log2_scale,log2_data,log2_lam", [(-600, -400, 300), (600, 300, -500), (-200, -700, 500), (0, -700, 0)])
def test_scales_with_blocks_apart(m, nv, log2_scale, log2_data, log2_lam):
    """A constant with a little noise, whose blocks take exponents of their own, small and with a scale far from 1."""
    rng = np.random.Generator(np.random.SFC64(m))
    n = 1 << m
    z = np.ldexp(1 + 1e-9 * rng.standard_normal((nv, n)), log2_data)
    scale, lam = 2.0 ** log2_scale, np.full(n, 2.0 ** log2_lam)
    x, xr, xi = z.copy(), z.copy(), np.zeros_like(z)
    tc_fft.fwht_mul_fwht(nv, 1, n // 2, lam, x, scale=scale)
    tc_fft.fft_mul_ifft(nv, 1, n // 2, lam, np.zeros(n), xr, xi, scale=scale)
    back = -(log2_scale + log2_lam)
    for y in (x, xr):
        # halves of the way back: the whole factor need not be a double
        y = np.ldexp(np.ldexp(y, back // 2 - log2_data // 2), back - back // 2 - (log2_data - log2_data // 2))
        one = np.ldexp(z, -log2_data)
        assert np.abs(y - one).max() < 4e-15
