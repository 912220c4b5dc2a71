"""The tensor-core kernel product where lam is applied as the accumulators are read (index bits of the last
forward pass a multiple of four) and where it is not, with tiles that end beyond the data."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,vectors", [(3, 5), (4, 300), (4, 257), (8, 17), (8, 1), (9, 9), (12, 3), (15, 2), (16, 3)])
@pytest.mark.parametrize("per_element,divide", [(False, False), (True, False), (False, True), (True, True)])
def test_product(m, vectors, per_element, divide):
    from qmctoolscl_gb300 import tc_fft
    rng = np.random.Generator(np.random.SFC64(40 + m))
    n = 1 << m
    br = np.array([int(format(i, "0%db" % m)[::-1], 2) for i in range(n)])
    y = rng.standard_normal((vectors, n)) + 1j * rng.standard_normal((vectors, n))
    lam = (0.5 + rng.random((vectors, n) if per_element else n)) * \
        np.exp(2j * np.pi * rng.random((vectors, n) if per_element else n))
    Y = np.fft.fft(y[:, br], norm="ortho")
    want = np.fft.ifft(Y / lam if divide else Y * lam, norm="ortho")[:, br]
    xr, xi = np.ascontiguousarray(y.real), np.ascontiguousarray(y.imag)
    tc_fft.fft_mul_ifft_tc(vectors, 1, n // 2, np.ascontiguousarray(lam.real), np.ascontiguousarray(lam.imag), xr, xi,
                           divide=divide)
    err = np.linalg.norm((xr + 1j * xi) - want, axis=1) / np.linalg.norm(want, axis=1)
    assert err.max() < 1e-6, err.max()
