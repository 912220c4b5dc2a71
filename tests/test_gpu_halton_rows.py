"""The fused Halton plan on its shared-memory tables (plans of a few million coordinates and more) against the
same plan on the warp kernel (any split of the adds selects it; that kernel is held to the oracle in
test_gpu_halton.py), bit for bit over the whole output: primes, composite and power-of-two bases (ties in
every row), large bases (groups of fewer dimensions), matrices without an inverse, every set of steps,
digits beyond their base, odd sizes and starts, few digits, and a batch."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PRIMES = [p for p in range(2, 542) if all(p % q for q in range(2, int(p ** 0.5) + 1))]


def _dims(rng, r, n_last, bases, lms, perm, shift, tmax=None, wide=False):
    import torch
    dims = []
    for b in bases:
        t = tmax or math.ceil(64 / math.log2(b))
        mmax, v = 0, n_last
        while v:
            v //= b
            mmax += 1
        C = np.zeros((mmax, t), np.int64)
        for k in range(min(mmax, t)):
            C[k, k] = 1
        q = dict(b=b, tmax=t, mmax=mmax, C=C)
        if lms:
            q["S"] = np.tril(rng.integers(0, b, (r, t, t)), -1) + np.eye(t, dtype=np.int64)
        if perm:
            q["perms"] = rng.random((r, t, b)).argsort(axis=2) + (3 * b if wide else 0)
        if shift:
            q["shifts"] = rng.integers(0, b, (r, t))
        dims.append({k: torch.from_numpy(np.ascontiguousarray(v)).cuda() if isinstance(v, np.ndarray) else v
                     for k, v in q.items()})
    return dims


def _both(plan, outs):
    import torch
    for x in outs:
        x.fill_(-1.0)
    plan.prepare()
    plan.run()
    got = [x.clone() for x in outs]
    plan.set_fp64_share(0.5)  # the warp kernel
    for x in outs:
        x.fill_(-2.0)
    plan.run()
    torch.cuda.synchronize()
    for a, x in zip(got, outs):
        assert torch.equal(a.view(torch.int64), x.view(torch.int64))
    assert all((a >= 0).all() for a in got)


CASES = [  # r, n, n_start, bases, lms, perm, shift, tmax
    (1, 1 << 18, 0, PRIMES, True, True, True, None),
    (2, 130001, 12345, PRIMES[:97], True, True, False, None),
    (1, 300000, (1 << 31) + 7, PRIMES[:83], True, False, True, None),
    (1, 400000, 1, PRIMES[:61], False, False, True, None),
    (1, 400000, 0, PRIMES[:61], False, True, False, None),
    (1, 400000, 0, PRIMES[:61], True, False, False, 9),
    (3, 200000, 5, [2, 4, 6, 8, 9, 10, 12, 15, 16, 25, 27, 32, 33, 36, 49, 64, 81, 100, 121, 128, 169, 256, 243, 512,
                    255, 30, 31, 1024, 35, 77, 91, 500, 60, 62, 2, 16, 48, 3, 5, 7, 256], True, True, True, None),
    (1, 1700000, 0, [2047, 2039, 1024, 1999, 2, 1500, 1733, 3, 1021, 997, 2000, 1900, 1013, 5, 1801], True, True, True, None),
]


@pytest.mark.parametrize("r,n,n_start,bases,lms,perm,shift,tmax", CASES)
def test_tables_equal_the_warp_kernel(r, n, n_start, bases, lms, perm, shift, tmax):
    import torch
    from qmctoolscl_gb300 import halton
    rng = np.random.Generator(np.random.SFC64(n + len(bases)))
    assert r * n * len(bases) >= 2.4e7
    x = torch.empty((r, n, len(bases)), dtype=torch.float64, device="cuda")
    _both(halton.HaltonPlan(r, n, n_start, _dims(rng, r, n_start + n - 1, bases, lms, perm, shift, tmax), x), [x])


def test_digits_beyond_their_base():
    import torch
    from qmctoolscl_gb300 import halton
    rng = np.random.Generator(np.random.SFC64(8))
    n, bases = 500000, PRIMES[:50]
    x = torch.empty((1, n, 50), dtype=torch.float64, device="cuda")
    _both(halton.HaltonPlan(1, n, 0, _dims(rng, 1, n - 1, bases, True, True, False, wide=True), x), [x])


def test_batch_and_graph():
    import torch
    from qmctoolscl_gb300 import halton
    rng = np.random.Generator(np.random.SFC64(9))
    reqs, outs = [], []
    for r, n, d in ((2, 65536, 100), (1, 20011, 37), (3, 99999, 21), (1, 262144, 27), (1, 7, 3)):
        x = torch.empty((r, n, d), dtype=torch.float64, device="cuda")
        reqs.append(dict(r=r, n=n, n_start=3 * d, dims=_dims(rng, r, 3 * d + n - 1, PRIMES[:d], True, True, True), x=x))
        outs.append(x)
    plan = halton.HaltonBatch(reqs)
    assert plan.coords >= 2.4e7
    s = torch.cuda.Stream()
    plan.graph_launch(s)
    s.synchronize()
    first = [x.clone() for x in outs]
    _both(plan, outs)
    assert all(torch.equal(a, x) for a, x in zip(first, outs))


def test_largest_digits():
    # point 0 has the largest digit everywhere: sums that round up to 1 in power-of-two bases
    import torch
    from qmctoolscl_gb300 import halton
    n, bases = 800000, [2, 4, 16, 256, 8, 32, 64, 128, 512, 1024, 2, 3, 5, 7, 31, 541] * 2
    rng = np.random.Generator(np.random.SFC64(10))
    dims = _dims(rng, 1, n - 1, bases, False, False, True)
    for q in dims:
        q["shifts"].fill_(q["b"] - 1)
    x = torch.empty((1, n, len(bases)), dtype=torch.float64, device="cuda")
    _both(halton.HaltonPlan(1, n, 0, dims, x), [x])
    assert float(x[0, 0, 0]) == 1.0


@pytest.mark.parametrize("r,n,n_start,bases", [(16, (1 << 20) + 777, 0, [2, 3, 5, 7, 29, 31, 37, 101, 541, 547]),
                                               (40, 300001, 1 << 20, [2, 4, 6, 9, 16, 25, 36, 64, 97, 211, 256, 540])])
def test_sections(r, n, n_start, bases):
    """Plans of 120 million coordinates and more, where a CTA's points come in several sections: sections
    that end early and last CTAs with part of their points."""
    import torch
    from qmctoolscl_gb300 import halton
    rng = np.random.Generator(np.random.SFC64(n))
    x = torch.empty((r, n, len(bases)), dtype=torch.float64, device="cuda")
    _both(halton.HaltonPlan(r, n, n_start, _dims(rng, r, n_start + n - 1, bases, True, True, True), x), [x])


@pytest.mark.parametrize("r,n,n_start,bases", [(1, 1000003, 0, [2, 3, 5]), (64, 4097, 65535, [2, 3, 7, 37, 53, 101, 541, 9, 4, 25]),
                                               (3, 40000, 99, PRIMES[:21]), (150, 4001, 0, [31, 29, 2, 547, 64])])
def test_smallest_plans(r, n, n_start, bases):
    """Plans of a few million coordinates: two steps of points per CTA."""
    import torch
    from qmctoolscl_gb300 import halton
    rng = np.random.Generator(np.random.SFC64(n))
    x = torch.empty((r, n, len(bases)), dtype=torch.float64, device="cuda")
    _both(halton.HaltonPlan(r, n, n_start, _dims(rng, r, n_start + n - 1, bases, True, True, True), x), [x])


@pytest.mark.parametrize("r,n,d", [(2, 130001, 12), (1, 262144, 21)])
def test_pinned_output(r, n, d):
    """Outputs in pinned host memory, which keep the warp kernel."""
    import torch
    from qmctoolscl_gb300 import batch, halton
    rng = np.random.Generator(np.random.SFC64(n))
    dims = _dims(rng, r, n - 1, PRIMES[:d], True, True, True)
    x = torch.empty((r, n, d), dtype=torch.float64, device="cuda")
    host = batch.pinned_empty((r, n, d))
    for out in (x, host):
        plan = halton.HaltonPlan(r, n, 0, dims, out)
        plan.prepare()
        plan.run()
    torch.cuda.synchronize()
    assert np.array_equal(x.cpu().numpy(), host)
