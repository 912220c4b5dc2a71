"""The FP64 transforms' block fixed-point passes against numpy: every split into a low pass of 9 to 12 bits
and high passes of 8 and 4, the FP64 kernel at the lengths and counts that keep it, and tiles that
must take the FP64 stages (zeros, inf, nan, values near the ends of the exponent range).  The
tolerance is per vector, 2e-15 relative L2: numpy's and the FP64 stages' own errors are 2 to 4e-16
up to 2^21."""
import numpy as np
import pytest

import qmctoolscl_gb300 as q
from qmctoolscl_gb300 import tc_fft

pytestmark = pytest.mark.gpu
U = np.uint64
TOL = 2e-15


def _bitrev(m):
    i = np.arange(1 << m)
    out = np.zeros_like(i)
    for b in range(m):
        out |= ((i >> b) & 1) << (m - 1 - b)
    return out


def _fwht(x):
    n, h = x.shape[-1], 1
    y = x.copy()
    while h < n:
        v = y.reshape(-1, n // (2 * h), 2, h)
        y = np.stack((v[:, :, 0] + v[:, :, 1], v[:, :, 0] - v[:, :, 1]), axis=2).reshape(-1, n)
        h *= 2
    return y / np.sqrt(n)


def _run(z, m):
    nv, n = z.shape
    tw = np.empty(n), np.empty(n)
    f, g = [z.real.copy(), z.imag.copy()], [z.real.copy(), z.imag.copy()]
    w = z.real.copy()
    q.fft_bro_1d_radix2(U(nv), U(1), U(n // 2), *tw, *f)
    q.ifft_bro_1d_radix2(U(nv), U(1), U(n // 2), *tw, *g)
    q.fwht_1d_radix2(U(nv), U(1), U(n // 2), w)
    return f[0] + 1j * f[1], g[0] + 1j * g[1], w


def _close(got, want):
    unit = np.maximum(np.abs(want).max(axis=1, keepdims=True), 1e-300)  # squares stay in range
    got, want = got / unit, want / unit
    err = np.linalg.norm(got - want, axis=1) / np.maximum(np.linalg.norm(want, axis=1), 1e-300)
    assert err.max() < TOL, err


@pytest.mark.parametrize("m,nv", [(8, 5), (9, 3), (9, 200), (10, 7), (11, 5), (12, 3), (13, 2), (14, 3), (15, 1),
                                  (16, 2), (17, 1), (18, 1), (19, 1), (20, 1), (21, 1), (10, 1700)])
def test_lengths(m, nv):
    rng = np.random.Generator(np.random.SFC64(m * 100 + nv))
    n = 1 << m
    z = rng.standard_normal((nv, n)) + 1j * rng.standard_normal((nv, n))
    z *= 10.0 ** rng.integers(-150, 150, (nv, 1))  # every vector at a scale of its own
    br = _bitrev(m)
    f, g, w = _run(z, m)
    _close(f, np.fft.fft(z[:, br], norm="ortho"))
    _close(g, np.fft.ifft(z, norm="ortho")[:, br])
    _close(w, _fwht(z.real))


@pytest.mark.parametrize("m", [9, 10, 11, 12, 13, 16, 20])
def test_fused(m):
    rng = np.random.Generator(np.random.SFC64(m))
    n, nv = 1 << m, 2 if m > 9 else 160
    z = rng.standard_normal((nv, n)) + 1j * rng.standard_normal((nv, n))
    lam = 0.5 + rng.random(n) + 1j * rng.random(n)
    br = _bitrev(m)
    for divide in (False, True):
        y = np.fft.fft(z[:, br], norm="ortho")
        want = np.fft.ifft(y / lam if divide else y * lam, norm="ortho")[:, br] * 1.5
        xr, xi = z.real.copy(), z.imag.copy()
        tc_fft.fft_mul_ifft(nv, 1, n // 2, lam.real.copy(), lam.imag.copy(), xr, xi, divide=divide, scale=1.5)
        _close(xr + 1j * xi, want)
        w = _fwht(z.real)
        x = z.real.copy()
        tc_fft.fwht_mul_fwht(nv, 1, n // 2, lam.real.copy(), x, divide=divide)
        _close(x, _fwht(w / lam.real if divide else w * lam.real))


@pytest.mark.parametrize("m", [9, 12, 13, 17])
def test_special_tiles(m):
    rng = np.random.Generator(np.random.SFC64(m + 7))
    n, nv = 1 << m, 160
    z = rng.standard_normal((nv, n)) + 1j * rng.standard_normal((nv, n))
    z[0] = 0
    z[1] *= 1e-290
    z[2] *= 1e290
    z[3] = 1  # all in one output
    z[4] = 0
    z[4, n // 3] = 0.1  # an impulse
    z[5, n // 2] = np.nan
    z[6, 5] = np.inf
    z[7, : n // 2] = 0
    br = _bitrev(m)
    f, g, w = _run(z, m)
    keep = [k for k in range(12) if k not in (5, 6)] + [nv - 1]
    _close(f[keep], np.fft.fft(z[keep][:, br], norm="ortho"))
    _close(g[keep], np.fft.ifft(z[keep], norm="ortho")[:, br])
    _close(w[keep], _fwht(z[keep].real))
    for y in (f, g, w):
        assert np.isfinite(y[[k for k in range(nv) if k not in (5, 6)]]).all()
        assert np.isnan(y[5]).all() and not np.isfinite(y[6]).any()
    assert not f[0].any() and not g[0].any() and not w[0].any()
