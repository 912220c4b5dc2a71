"""Lattice shifts off the 2^-53 grid (torch.rand on the GPU draws odd multiples of 2^-54) against the
oracle, bit for bit: the fused kernel, the batched plan and the plain mod-1 shift, over even and odd
dimensions and shifts that make ties, sums of 1 and of 2, and results below 2^-32."""
import numpy as np
import pytest

import oracle
import qmctoolscl_gb300 as q
from qmctoolscl_gb300 import batch

pytestmark = pytest.mark.gpu
U = np.uint64


def _shifts(kind, rng, r, d):
    if kind == "half_grid":  # odd multiples of 2^-54
        s = rng.integers(0, 1 << 53, (r, d)).astype(np.float64) * 2.0 ** -53
        return np.where(s < 0.5, s + 2.0 ** -54, s)
    if kind == "tiny":  # multiples of 2^-64 below 2^-11
        return rng.integers(0, 1 << 53, (r, d)).astype(np.float64) * 2.0 ** -64
    s = 2.0 ** -rng.integers(1, 64, (r, d)).astype(np.float64)  # edges: one bit, its complement, nearly 1
    s[:, 1::3] = 1 - 2.0 ** -rng.integers(1, 54, (r, d)).astype(np.float64)[:, 1::3]
    s[:, 2::3] = 2.0 ** -64 * rng.integers(1, 4, (r, d))[:, 2::3]
    return s


@pytest.mark.parametrize("kind", ["half_grid", "tiny", "edges"])
@pytest.mark.parametrize("order,n,d", [("gray", 1000, 7), ("natural", 1 << 12, 64), ("gray", 1, 2), ("gray", 33, 1)])
def test_shift_off_the_grid(kind, order, n, d):
    import torch
    rng = np.random.Generator(np.random.SFC64(n + d))
    r = 3
    g = rng.integers(0, 1 << 19, (r, d)).astype(U) * U(2) + U(1)
    s = _shifts(kind, rng, r, d)
    x, want = np.empty((r, n, d)), np.empty((r, n, d))
    oracle.call("lat_gen_" + order, U(r), U(n), U(d), U(0), g, x)
    oracle.call("lat_shift_mod_1", U(r), U(n), U(d), U(r), x, s, want)
    gt, st = torch.from_numpy(g.view(np.int64)).cuda(), torch.from_numpy(s).cuda()
    got = [torch.full((r, n, d), -1.0, dtype=torch.float64, device="cuda") for _ in range(3)]
    batch.lattice_gen_shift(r, n, d, 0, gt, st, got[0], order=order)
    batch.LatPlan([dict(r=r, n=n, d=d, order=order, g=gt, shifts=st, x=got[1])]).run()
    q.lat_shift_mod_1(U(r), U(n), U(d), U(r), torch.from_numpy(x).cuda(), st, got[2])
    for y in got:
        assert np.array_equal(y.cpu().numpy().view(U), want.view(U))
