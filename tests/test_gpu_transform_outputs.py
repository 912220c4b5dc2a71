"""The FP64 transforms output by output: relative errors against long double on data whose transform is not alike
in size (a constant with a little noise, products, kernel columns of lattices and nets), no larger
than those of the same stages in float64 (numpy, radix 2).  Compared are the L2 error, the median and
the 90th percentile of |error| / |output|: at most twice the float64 stages' plus 3e-16 (two roundings of a
result).  Further: whole numbers exactly, blocks of far different size and of zeros in one tile, and products
that leave the fixed-point range after the pointwise step."""
import numpy as np
import pytest

import qmctoolscl_gb300 as q
from qmctoolscl_gb300 import tc_fft

pytestmark = pytest.mark.gpu
U, L = np.uint64, np.longdouble
PI = L("3.14159265358979323846264338327950288")


def bitrev(m):
    i = np.arange(1 << m)
    out = np.zeros_like(i)
    for b in range(m):
        out |= ((i >> b) & 1) << (m - 1 - b)
    return out


def wht(x, t):
    n, h, y = x.shape[-1], 1, x.astype(t)
    while h < n:
        v = y.reshape(-1, n // (2 * h), 2, h)
        y = np.stack((v[:, :, 0] + v[:, :, 1], v[:, :, 0] - v[:, :, 1]), axis=2).reshape(x.shape)
        h *= 2
    return y / np.sqrt(t(n))


def dft(x, t, inverse=False):
    """bit-reversed input of a real array, natural output, orthonormal, in type t: (real, imaginary)"""
    n = x.shape[-1]
    r, i = x.astype(t), np.zeros(x.shape, t)
    h = 1
    while h < n:
        a = PI * np.arange(h, dtype=L) / h
        c, s = np.cos(a).astype(t), (np.sin(a) if inverse else -np.sin(a)).astype(t)
        r, i = r.reshape(-1, n // (2 * h), 2, h), i.reshape(-1, n // (2 * h), 2, h)
        tr, ti = r[:, :, 1] * c - i[:, :, 1] * s, r[:, :, 1] * s + i[:, :, 1] * c
        r, i = np.stack((r[:, :, 0] + tr, r[:, :, 0] - tr), axis=2), np.stack((i[:, :, 0] + ti, i[:, :, 0] - ti), axis=2)
        h *= 2
    f = 1 / np.sqrt(t(n))
    return r.reshape(x.shape) * f, i.reshape(x.shape) * f


def _product(v, m):
    x = np.ones(1)
    for _ in range(m):
        x = np.concatenate((x, x * v))
    return x


def _net(m, d, rng):
    i, X = np.arange(1 << m, dtype=U), np.zeros((1 << m, d), U)
    for j in range(d):
        for k in range(m):
            above = (int(rng.integers(0, 1 << 32)) >> (32 - k)) << (32 - k) if j and k else 0
            X[:, j] ^= U(above | 1 << (31 - k)) * ((i >> U(k)) & U(1))
    return X / 2.0 ** 32


def _walsh_kernel(m, d, rng):
    """first column of a digitally shift invariant kernel matrix (order 2) on a net"""
    X = _net(m, d, rng)
    b = -np.floor(np.log2(np.where(X > 0, X, 1.0)))
    return np.prod(1 + np.where(X > 0, -b * X + 2.5 * (1 - 2.0 ** -b), 2.5), axis=1)


def _lattice_kernel(m, d, order):
    n = 1 << m
    x = (np.arange(n)[:, None] * np.array([1, 182667, 469891, 498753][:d]) % n) / n
    k = 2 * np.pi ** 2 * (x * x - x + 1 / 6) if order == 2 else \
        -(2 * np.pi) ** 4 / 24 * (x ** 4 - 2 * x ** 3 + x * x - 1 / 30)
    return np.prod(1 + k, axis=1)


def data(m):
    n, rng, br = 1 << m, np.random.Generator(np.random.PCG64(m)), bitrev(m)
    one = np.ones(n)
    one[n // 3] = 1 + 2.0 ** -50
    t = np.arange(n) / n
    return {"normal": rng.standard_normal(n), "lognormal": np.exp(3 * rng.standard_normal(n)),
            "16 decades": 10.0 ** rng.uniform(-16, 0, n), "whole": 1e12 + rng.integers(-1000, 1000, n), "one differs": one,
            "1 + 1e-12 noise": 1 + 1e-12 * rng.standard_normal(n), "1 + 1e-6 noise": 1 + 1e-6 * rng.standard_normal(n),
            "alternating + noise": 1e6 * (-1.0) ** np.arange(n) + rng.standard_normal(n),
            "[1, .99]": _product(0.99, m), "[1, .999]": _product(0.999, m), "[1, .5]": _product(0.5, m),
            "walsh 1": _walsh_kernel(m, 1, rng), "walsh 4": _walsh_kernel(m, 4, rng),
            "smooth": np.exp(np.cos(2 * np.pi * t))[br], "bump": np.exp(-50 * (t - 0.5) ** 2)[br],
            "lattice 1": _lattice_kernel(m, 1, 2)[br], "lattice 3": _lattice_kernel(m, 3, 4)[br]}


def _errors(got, want):
    e, w = np.abs(got - want), np.abs(want)
    rel = (e[w > 0] / w[w > 0]).astype(float)
    return float(np.sqrt((e * e).sum() / (w * w).sum())), float(np.median(rel)), float(np.quantile(rel, 0.9))


def _no_worse(got, stages, want, what):
    g, s = _errors(got, want), _errors(stages, want)
    assert all(a <= 2 * b + 3e-16 for a, b in zip(g, s)), (what, g, s)


@pytest.mark.parametrize("m,copies", [(9, 10), (10, 1), (11, 1), (12, 1), (13, 1), (15, 1), (16, 1)])
def test_small_outputs(m, copies):
    S = data(m)
    n, br = 1 << m, bitrev(m)
    X = np.stack(list(S.values()))
    big = np.tile(X, (copies, 1))
    nv = len(big)
    tw = np.empty(n), np.empty(n)
    w, f, fi, g, gi = big.copy(), big.copy(), np.zeros_like(big), big[:, br].copy(), np.zeros_like(big)
    q.fwht_1d_radix2(U(nv), U(1), U(n // 2), w)
    q.fft_bro_1d_radix2(U(nv), U(1), U(n // 2), *tw, f, fi)
    q.ifft_bro_1d_radix2(U(nv), U(1), U(n // 2), *tw, g, gi)
    W, W64, F, F64, G, G64 = wht(X, L), wht(X, np.float64), dft(X, L), dft(X, np.float64), dft(X, L, True), dft(X, np.float64, True)
    both = lambda r, i: np.stack((r, i)).astype(L)  # noqa: E731
    for k, name in enumerate(S):
        _no_worse(w[k].astype(L), W64[k].astype(L), W[k], ("wht", name))
        _no_worse(both(f[k], fi[k]), both(F64[0][k], F64[1][k]), both(F[0][k], F[1][k]), ("fft", name))
        _no_worse(both(g[k], gi[k]), both(G64[0][k][br], G64[1][k][br]), both(G[0][k][br], G[1][k][br]), ("ifft", name))
    assert np.array_equal(w[:len(X)], w[-len(X):]) and np.array_equal(f[:len(X)], f[-len(X):])


@pytest.mark.parametrize("m,nv", [(10, 3), (12, 2), (16, 1), (20, 1)])
def test_whole_numbers_exactly(m, nv):
    """Sums of whole numbers below 2^53 in all: the Walsh-Hadamard transform of an even number of stages is exact."""
    rng = np.random.Generator(np.random.SFC64(m))
    n = 1 << m
    x = rng.integers(-(1 << (52 - m)), 1 << (52 - m), (nv, n)).astype(np.float64)
    x[0, : n // 2] = 1 << (52 - m)  # and small ones beside large sums
    want = np.rint(wht(x, np.float64) * np.sqrt(float(n))) / np.sqrt(float(n))
    q.fwht_1d_radix2(U(nv), U(1), U(n // 2), x)
    assert np.array_equal(x, want)


@pytest.mark.parametrize("m,nv", [(9, 200), (10, 4), (11, 4), (12, 4), (13, 4), (16, 4), (17, 2)])
def test_blocks_apart(m, nv):
    """Sixteen consecutive or strided values alone in their size, from next to nothing to next to everything, and zeros
    about them: L2 errors within 2e-15 as elsewhere, and nothing that is zero moves."""
    rng = np.random.Generator(np.random.SFC64(m))
    n, br = 1 << m, bitrev(m)
    x = np.zeros((nv, n))
    x[0, 16:32] = rng.standard_normal(16)
    x[0, 48:64] = 1e-200 * rng.standard_normal(16)
    x[1, :: n // 16] = rng.standard_normal(16)
    x[1, 1 :: n // 16] = 1e-290 * rng.standard_normal(16)
    if nv > 2:
        x[2] = rng.standard_normal(n)
        x[2, 64:128] *= 1e-30
        x[3, 5] = 1e-240
        x[3, 7] = -1e-240
        x[3, 6] = 1e-252
    tw = np.empty(n), np.empty(n)
    w, f, fi, g, gi = x.copy(), x.copy(), np.zeros_like(x), x.copy(), np.zeros_like(x)
    q.fwht_1d_radix2(U(nv), U(1), U(n // 2), w)
    q.fft_bro_1d_radix2(U(nv), U(1), U(n // 2), *tw, f, fi)
    q.ifft_bro_1d_radix2(U(nv), U(1), U(n // 2), *tw, g, gi)
    F, G = dft(x, L), dft(x[:, br], L, True)
    for got, want in ((w, wht(x, L)), (np.stack((f, fi), 1), np.stack(F, 1)), (np.stack((g, gi), 1), np.stack((G[0][:, br], G[1][:, br]), 1))):
        for k in range(min(nv, 4)):
            top = np.abs(want[k]).max()
            e = np.sqrt((((got[k] - want[k]) / top) ** 2).sum() / ((want[k] / top) ** 2).sum())
            assert e < 2e-15, (k, e)
        assert not got[4:].any()


@pytest.mark.parametrize("m", [9, 10, 12, 13, 16, 17])
@pytest.mark.parametrize("divide", [False, True])
def test_products_out_of_range(m, divide):
    """lam of its own for every vector: zeros, infinities, NaN and numbers that take a product out of the fixed-point
    range spoil (or scale) their own vector only."""
    rng = np.random.Generator(np.random.SFC64(m))
    n, nv = 1 << m, 160 if m == 9 else 8
    x = rng.standard_normal((nv, n))
    lam = 0.5 + rng.random((nv, n))
    lam[1, n // 2] = np.inf
    lam[2, 3] = np.nan
    lam[3, 7] = 0.0
    lam[4] = 1e-290 if not divide else 1e290 ** 0.5
    lam[5] *= 10.0 ** rng.uniform(-40, 0, n)
    lam[6] = 2.0 ** -500 if divide else 2.0 ** 500
    lr = lam.copy()
    a, b, bi = x.copy(), x.copy(), np.zeros_like(x)
    with np.errstate(all="ignore"):
        tc_fft.fwht_mul_fwht(nv, 1, n // 2, lr, a, divide=divide)
        tc_fft.fft_mul_ifft(nv, 1, n // 2, lr, np.zeros_like(lam), b, bi, divide=divide)
        y, z = wht(x, L), dft(x, L)
        want = wht(y / lam if divide else y * lam, L)
        br = bitrev(m)
        p = (z[0] / lam if divide else z[0] * lam), (z[1] / lam if divide else z[1] * lam)
        c, d = dft(p[0][:, br], L, True), dft(p[1][:, br], L, True)  # of the real and the imaginary part
        want_c = np.stack(((c[0] - d[1])[:, br], (c[1] + d[0])[:, br]), 1)
    got_c = np.stack((b, bi), 1)
    spoilt = {2} | ({3} if divide else {1})
    for got, ref in ((a, want), (got_c, want_c)):
        for k in range(8):
            if k in spoilt:
                assert not np.isfinite(got[k]).all()
                continue
            if k == 1 or (k == 4 and divide):
                continue  # 1 / inf; 1e145^2 in the complex quotient
            top = np.abs(ref[k]).max()
            e = np.sqrt((((got[k] - ref[k]) / top) ** 2).sum() / ((ref[k] / top) ** 2).sum())
            assert e < 2e-15, (k, float(e))
