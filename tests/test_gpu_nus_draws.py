"""The nested uniform scramble's draws against the oracle (outputs and generator states) where full and half
draws mix: widths on both sides of 32 bits, kept halves at the start, points at the ends of the 256-point
tiles and 32-output blocks, more than 32 generators, continuation calls, runs of repeated keys (no draws)."""
import numpy as np
import pytest

from .test_gpu_nus import _check_against_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tmax_new", [20, 33, 34, 43, 50, 64])
@pytest.mark.parametrize("n,r,d", [(1023, 1, 2), (255, 2, 3), (1024, 2, 3), (3000, 1, 3), (31, 5, 9), (32, 1, 1), (70000, 1, 2)])
def test_mixed_widths(tmax_new, n, r, d):
    rng = np.random.Generator(np.random.SFC64(n + tmax_new))
    mk = lambda: rng.integers(0, 1 << 62, (1, n, d), dtype=np.uint64) >> np.uint64(62 - min(tmax_new, 60))  # noqa: E731
    a, b = mk(), mk()
    a[:, n // 3: n // 2] = a[:, :1]  # repeats
    b[:, ::5] = a[:, ::5]
    _check_against_oracle(rng, r, n, d, 1, min(tmax_new, 60), tmax_new, [a, b])


@pytest.mark.parametrize("share", [2, 3, 7])
def test_sparse_half_draws(share):
    # pairs that share all but a few bits: one half draw in `share` points, tiles with none, one and two
    rng = np.random.Generator(np.random.SFC64(share))
    n = 9000
    xb = rng.integers(0, 1 << 63, (1, n, 2), dtype=np.uint64) * np.uint64(2)
    close = np.arange(1, n) % (share * 300) < share
    xb[:, 1:][:, close] = xb[:, :-1][:, close] ^ np.uint64(1 << 20)
    _check_against_oracle(rng, 1, n, 2, 1, 64, 64, [xb, xb[:, ::-1].copy()])
