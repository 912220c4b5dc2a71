"""Which of its two generation kernels a Halton plan takes, on both sides of every limit of the rule; the table
kernel against the oracle itself; and a preparation captured in a CUDA graph that serves both kernels."""
import numpy as np
import pytest

from .test_gpu_halton import oracle_chain, same_bits
from .test_gpu_halton_rows import PRIMES, _dims

pytestmark = pytest.mark.gpu
U = np.uint64


def _plan(r, n, bases, x=None, n_start=0, **kw):
    import torch
    from qmctoolscl_gb300 import halton
    rng = np.random.Generator(np.random.SFC64(n + len(bases)))
    dims = _dims(rng, r, n_start + n - 1, bases, True, True, True, **kw)
    if x is None:
        x = torch.empty((r, n, len(bases)), dtype=torch.float64, device="cuda")
    return halton.HaltonPlan(r, n, n_start, dims, x), dims, x


# the plans that test_gpu_halton_rows compares, the smallest and the odd ones among them, and plans
# just below each limit (2.4 million coordinates, 4000 points per randomisation)
@pytest.mark.parametrize("r,n,bases,tables", [
    (1, 1000003, [2, 3, 5], True), (64, 4097, [2, 3, 7, 37, 53, 101, 541, 9, 4, 25], True), (3, 40000, PRIMES[:21], True),
    (150, 4001, [31, 29, 2, 547, 64], True), (1, 1700000, [2047, 2039, 1024, 1999, 2], True), (2, 130001, PRIMES[:97], True),
    (16, (1 << 20) + 777, [2, 3, 5, 7, 29, 31, 37, 101, 541, 547], True),
    (1, 799999, [2, 3, 5], False), (151, 3999, [31, 29, 2, 547, 64], False), (1, 1000, PRIMES[:10], False)])
def test_rule(r, n, bases, tables):
    plan, _, _ = _plan(r, n, bases)
    assert plan.info() == {"has_tables": tables, "uses_tables": tables}
    plan.set_fp64_share(0.5)
    assert plan.info() == {"has_tables": tables, "uses_tables": False}
    plan.set_fp64_share(1.0)
    assert plan.info() == {"has_tables": tables, "uses_tables": tables}


@pytest.mark.parametrize("b", [2, 3, 4, 5, 8, 16, 25, 31, 32, 37, 64, 101, 128, 211, 256, 509])
def test_one_dimension(b):
    """Plans of one dimension, small tables: some of them fit the 48 KB that a kernel has unasked only without the
    kernel's static arrays."""
    import torch
    plan, _, x = _plan(1, 2400007, [b])
    assert plan.info()["uses_tables"]
    plan.prepare()
    plan.run()
    torch.cuda.synchronize()
    got = x.clone()
    plan.set_fp64_share(0.5)
    x.fill_(-1.0)
    plan.run()
    torch.cuda.synchronize()
    assert torch.equal(x.view(torch.int64), got.view(torch.int64))


def test_pinned_output_has_no_tables():
    from qmctoolscl_gb300 import batch
    plan, _, _ = _plan(2, 130001, PRIMES[:12], batch.pinned_empty((2, 130001, 12)))
    assert plan.info() == {"has_tables": False, "uses_tables": False}


@pytest.mark.parametrize("r,n,n_start,bases", [(1, 810001, 0, [2, 3, 541]), (2, 60001, 1 << 30, PRIMES[:21])])
def test_tables_against_oracle(r, n, n_start, bases):
    """Every dimension's chain of plain calls on its first, middle and last points."""
    plan, dims, x = _plan(r, n, bases, n_start=n_start)
    assert plan.info()["uses_tables"]
    plan.prepare()
    plan.run()
    got = x.cpu().numpy()
    host = [{k: np.ascontiguousarray(v.cpu().numpy()).view(U) if hasattr(v, "cpu") else v for k, v in q.items()} for q in dims]
    for i0 in (0, n // 2 - 350, n - 700):
        assert same_bits(got[:, i0:i0 + 700], oracle_chain(r, 700, n_start + i0, host))


def test_captured_preparation_serves_both_kernels():
    """Rows of digits that are all zero between others: the warp kernel must not stop at them."""
    import torch
    plan, dims, x = _plan(1, 500000, [2, 3, 5, 7, 11])
    for q in dims:
        q["perms"][:, 4:12] = 0
        q["shifts"][:, 4:12] = 0
    assert plan.info()["uses_tables"]
    s = torch.cuda.Stream()
    plan.prepare(s)
    plan.run(s)
    s.synchronize()
    want = x.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        plan.prepare(s)
    plan.set_fp64_share(0.5)
    assert not plan.info()["uses_tables"]
    x.fill_(-1.0)
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    plan.run()
    torch.cuda.synchronize()
    assert torch.equal(x.view(torch.int64), want.view(torch.int64))
