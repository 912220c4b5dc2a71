"""halton_qrng's shared levels at the sizes where they can go wrong: ends of the 4096-point chunks, one
point, index ranges that start inside a block of every base or wrap to 0, top levels of one to 256
values, bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
from qmctoolscl_gb300.c_funcs import halton_qrng_c

pytestmark = pytest.mark.gpu

DIMS = np.array([0, 1, 2, 3, 5, 6, 17, 53, 54, 99, 200, 359], dtype=np.int32)


@pytest.mark.parametrize("gen", [0, 1])
@pytest.mark.parametrize("n,n0", [(1, 0), (4095, 0), (4096, 1), (4097, 4095), (8193, 65535), (70001, 2 ** 20 - 7),
                                  (5000, -4999), (5000, -1), (9000, 2 ** 31 - 9001)])
def test_chunks(n, n0, gen):
    rng = np.random.Generator(np.random.SFC64(n + gen))
    d = len(DIMS)
    randu = rng.random(d * 32)
    randu[:32] = 0.0  # no shifts: zero prefixes
    want, res = np.full(d * n, np.nan), np.full(d * n, np.nan)
    oracle.halton_qrng(n, d, n0, gen, want, randu, DIMS)
    halton_qrng_c(n, d, n0, gen, res, randu, DIMS)
    assert np.array_equal(want.view(np.uint64), res.view(np.uint64))
