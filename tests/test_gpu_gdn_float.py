"""gdn_integer_to_float where the sum runs in integers, against the oracle bit for bit: power-of-two bases
(ties and carries up to 1), small and large bases, digit counts around the sections' ends and the
eight-digit groups, all-zero, largest, leading-zero and out-of-range digits, odd dimensions."""
import numpy as np
import pytest

import oracle
import qmctoolscl_gb300 as q

pytestmark = pytest.mark.gpu
U = np.uint64


@pytest.mark.parametrize("bases", [[2], [2, 3, 5, 7], [4, 16, 8], [3, 31, 13, 2, 29], [541], [127], [64], [2, 2]])
@pytest.mark.parametrize("tmax", [1, 2, 7, 8, 13, 14, 16, 33, 54, 64])
def test_sections(bases, tmax):
    rng = np.random.Generator(np.random.SFC64(tmax * 1000 + sum(bases)))
    r, n, d = 2, 700, len(bases)
    b = np.array([bases], dtype=U)
    x = rng.integers(0, 1 << 40, (r, n, d, tmax), dtype=U) % b[0][None, None, :, None]
    x[:, 0] = 0
    x[:, 1] = b[0][None, :, None] - U(1)
    for i in range(40):  # zeros or largest digits first, then random, zero or largest ones
        t = int(rng.integers(0, tmax + 1))
        x[:, 2 + i, :, :t] = 0 if i % 2 else b[0][None, :, None] - U(1)
        if i % 3 == 0:
            x[:, 2 + i, :, t + 1:] = b[0][None, :, None] - U(1)
        if i % 3 == 1:
            x[:, 2 + i, :, t + 1:] = 0
    x[0, 50, :, tmax // 2] = b[0]
    x[0, 51, :, 0] = U(1 << 33)
    x[0, 52, :, tmax - 1] = U(5000)
    want, got = np.empty((r, n, d)), np.empty((r, n, d))
    oracle.call("gdn_integer_to_float", U(r), U(n), U(d), U(1), U(tmax), b, x, want)
    q.gdn_integer_to_float(U(r), U(n), U(d), U(1), U(tmax), b, x, got)
    assert np.array_equal(got.view(U), want.view(U))


@pytest.mark.parametrize("r, n, bases, tmax", [
    (1, 500009, [2], 16), (1, 470011, [2], 64), (3, 90001, [2, 3, 5, 7], 20), (2, 120007, [4, 16], 33),
    (1, 100003, [3, 31, 13, 2, 29], 23), (401, 4001, [2], 22), (400, 2111, [2, 5], 54), (1, 15013, [2] * 32, 32),
    (640, 4003, [541, 2], 16), (2, 20011, [2] * 50, 16)])
def test_large_calls(r, n, bases, tmax):
    """Sizes that go by staged digits, in one wave of blocks and in several, with all kinds of rows."""
    rng = np.random.Generator(np.random.SFC64(tmax * 1000 + sum(bases)))
    d = len(bases)
    b = np.array([bases], dtype=U)
    x = rng.integers(0, 1 << 40, (r, n, d, tmax), dtype=U) % b[0][None, None, :, None]
    for i in range(0, n, 31):  # zeros or largest digits first
        t = int(rng.integers(0, tmax + 1))
        x[:, i, :, :t] = 0 if i % 2 else b[0][None, :, None] - U(1)
    x[0, 50, :, tmax // 2] = b[0]
    x[0, 51, :, 0] = U(1 << 33)
    x[-1, -1, :, tmax - 1] = U(5000)
    want, got = np.empty((r, n, d)), np.empty((r, n, d))
    oracle.call("gdn_integer_to_float", U(r), U(n), U(d), U(1), U(tmax), b, x, want)
    q.gdn_integer_to_float(U(r), U(n), U(d), U(1), U(tmax), b, x, got)
    assert np.array_equal(got.view(U), want.view(U))
