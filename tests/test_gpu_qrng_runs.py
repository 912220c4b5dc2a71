"""halton_qrng's runs of points per warp at the sizes where they can go wrong: fewer points than a CTA's
warps, shares of a warp that end inside 32 points, several runs per warp in the small bases, and runs that
wrap to index 0, bit for bit against the oracle."""
import numpy as np
import pytest

import oracle
from qmctoolscl_gb300.c_funcs import halton_qrng_c

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [[0], [1, 4], [0, 2, 30, 359]])
@pytest.mark.parametrize("n,n0", [(31, 0), (33, 5), (225, 0), (257, 31), (1025, 1023), (2049, -1000), (12289, 2 ** 20),
                                  (400009, 12345), (300001, -150000), (65536, 2 ** 31 - 65537)])
def test_runs(n, n0, dims):
    rng = np.random.Generator(np.random.SFC64(n))
    dims = np.array(dims, dtype=np.int32)
    d = len(dims)
    randu = rng.random(d * 32)
    want, res = np.full(d * n, np.nan), np.full(d * n, np.nan)
    oracle.halton_qrng(n, d, n0, 1, want, randu, dims)
    halton_qrng_c(n, d, n0, 1, res, randu, dims)
    assert np.array_equal(want.view(np.uint64), res.view(np.uint64))
