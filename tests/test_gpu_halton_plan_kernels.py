"""A Halton plan's preparation captured in a CUDA graph serves both generation kernels."""
import numpy as np
import pytest

from .test_gpu_halton_rows import PRIMES, _dims

pytestmark = pytest.mark.gpu


def _plan(r, n, bases, x=None, n_start=0, **kw):
    import torch
    from qmctoolscl_gb300 import halton
    rng = np.random.Generator(np.random.SFC64(n + len(bases)))
    dims = _dims(rng, r, n_start + n - 1, bases, True, True, True, **kw)
    if x is None:
        x = torch.empty((r, n, len(bases)), dtype=torch.float64, device="cuda")
    return halton.HaltonPlan(r, n, n_start, dims, x), dims, x


def test_captured_preparation_serves_both_kernels():
    """Rows of digits that are all zero between others: the warp kernel must not stop at them."""
    import torch
    plan, dims, x = _plan(1, 500000, [2, 3, 5, 7, 11])
    for q in dims:
        q["perms"][:, 4:12] = 0
        q["shifts"][:, 4:12] = 0
    s = torch.cuda.Stream()
    plan.prepare(s)
    plan.run(s)
    s.synchronize()
    want = x.clone()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        plan.prepare(s)
    plan.set_fp64_share(0.5)
    x.fill_(-1.0)
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    plan.run()
    torch.cuda.synchronize()
    assert torch.equal(x.view(torch.int64), want.view(torch.int64))
