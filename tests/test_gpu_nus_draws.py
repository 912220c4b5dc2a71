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


@pytest.mark.parametrize("n", [63, 64, 65, 127, 129, 300, 20000])
def test_counters_near_their_upper_half(n):
    """Streams whose 64-bit counter carries into its upper half in, before and after a block of outputs."""
    import oracle
    import qmctoolscl_gb300 as q
    from .test_gpu_nus import _states
    rng = np.random.Generator(np.random.SFC64(n))
    d = 5
    gens = [np.random.Generator(np.random.SFC64(k)) for k in range(d)]
    for k, g in enumerate(gens):
        state = g.bit_generator.state
        state["state"]["state"][3] = np.uint64((1 << 32) * (k + 1) - (10, 64, 65, 200, 1)[k])
        g.bit_generator.state = state
    words = _states(gens).reshape(-1).copy()
    xb = rng.integers(0, 1 << 63, (1, n, d), dtype=np.uint64) * np.uint64(2)
    want, got = np.zeros((1, n, d), np.uint64), np.zeros((1, n, d), np.uint64)
    forest = oracle.NusForest(d)
    forest.scramble(1, n, d, 1, 64, 64, words, xb, want)
    roots = np.array([q.NUSNode_dnb2() for _ in range(d)]).reshape(1, d)
    q.dnb2_nested_uniform_scramble(1, n, d, 1, 64, 64, np.array(gens, dtype=object).reshape(1, d), roots, xb, got)
    forest.close()
    assert np.array_equal(got, want)
    assert np.array_equal(_states(gens).reshape(-1), words)


@pytest.mark.parametrize("d", [1, 10, 31, 32, 33, 37, 64, 70])
@pytest.mark.parametrize("n", [300, 700])
def test_generator_counts(d, n):
    """Generators that fill the streams' warps and that leave lanes without one, over several blocks of
    outputs, with counters that carry into their upper half at different blocks in different lanes, in one lane
    only, and in none."""
    import oracle
    import qmctoolscl_gb300 as q
    from .test_gpu_nus import _states
    rng = np.random.Generator(np.random.SFC64(n + d))
    gens = [np.random.Generator(np.random.SFC64(k)) for k in range(d)]
    for k, g in enumerate(gens):
        if k % 32 in (0, 5, 30) and k < 64:
            state = g.bit_generator.state
            state["state"]["state"][3] = np.uint64((1 << 32) * (k + 1) - (1 + 67 * (k % 32) // 5))
            g.bit_generator.state = state
    words = _states(gens).reshape(-1).copy()
    xb = rng.integers(0, 1 << 63, (1, n, d), dtype=np.uint64) * np.uint64(2)
    forest = oracle.NusForest(d)
    roots = np.array([q.NUSNode_dnb2() for _ in range(d)]).reshape(1, d)
    for part in (xb, xb[:, ::-1] ^ np.uint64(1 << 40)):
        want, got = np.zeros((1, n, d), np.uint64), np.zeros((1, n, d), np.uint64)
        part = np.ascontiguousarray(part)
        forest.scramble(1, n, d, 1, 64, 64, words, part, want)
        q.dnb2_nested_uniform_scramble(1, n, d, 1, 64, 64, np.array(gens, dtype=object).reshape(1, d), roots, part, got)
        assert np.array_equal(got, want)
        assert np.array_equal(_states(gens).reshape(-1), words)
    forest.close()
