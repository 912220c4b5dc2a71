"""Base-2 net kernels where they take new routes, against the oracle bit for bit: the shift and the float
conversion as runs of words (odd and uneven column counts, arrays 8 bytes off a 16-byte boundary, one of
the two off it, more columns than are staged, r_x < r), the index tables of every low-bit count and
column count, and the plans' matrix preparation (bit counts around 32 and 64, mmax above 32, alpha 1 to 5)."""
import numpy as np
import pytest

import oracle
import qmctoolscl_gb300 as q
from qmctoolscl_gb300 import batch

pytestmark = pytest.mark.gpu
U = np.uint64


def _cuda(a, off=0):
    """a copy on the GPU that starts `off` words after a 256-byte boundary"""
    import torch
    a = np.ascontiguousarray(a)
    t = torch.empty(a.size + off, dtype=torch.float64 if a.dtype == np.float64 else torch.int64, device="cuda")[off:]
    t.copy_(torch.from_numpy(a.reshape(-1).view(np.int64) if a.dtype == U else a.reshape(-1)))
    return t


def _bits(t):
    return t.cpu().numpy().view(U)


@pytest.mark.parametrize("r,r_x,n,d", [(2, 2, 20011, 5), (4, 2, 3001, 21), (1, 1, 70001, 3), (3, 1, 700, 127),
                                       (1, 1, 300000, 1), (2, 2, 64, 2050), (2, 2, 2000, 40)])
@pytest.mark.parametrize("off_in,off_out", [(0, 0), (1, 1), (0, 1), (1, 0)])
def test_runs(r, r_x, n, d, off_in, off_out):
    rng = np.random.Generator(np.random.SFC64(n + d))
    xb = rng.integers(0, 1 << 63, (r_x, n, d), dtype=U)
    sh, ls = rng.integers(0, 1 << 63, (r, d), dtype=U), rng.integers(0, 3, r_x, dtype=U)
    tm = rng.integers(50, 65, r, dtype=U)
    xrb, x = np.empty((r, n, d), U), np.empty((r, n, d))
    oracle.call("dnb2_digital_shift", U(r), U(n), U(d), U(r_x), ls, xb, sh, xrb)
    oracle.call("dnb2_integer_to_float", U(r), U(n), U(d), tm, xrb, x)
    got, gx = _cuda(np.zeros_like(xrb), off_out), _cuda(np.zeros_like(x), off_in)
    q.dnb2_digital_shift(U(r), U(n), U(d), U(r_x), _cuda(ls), _cuda(xb, off_in), _cuda(sh), got)
    assert np.array_equal(_bits(got), xrb.reshape(-1))
    q.dnb2_integer_to_float(U(r), U(n), U(d), _cuda(tm), got, gx)
    assert np.array_equal(_bits(gx), x.reshape(-1).view(U))


@pytest.mark.parametrize("r,r_x,n,d", [(1300, 1300, 199, 5), (1300, 1, 201, 5), (1300, 1300, 333, 6), (1300, 650, 334, 6),
                                       (1000, 1000, 49, 5), (1000, 1, 51, 5), (1000, 500, 83, 6), (1000, 2, 85, 6),
                                       (70000, 35000, 1, 3), (70000, 70000, 2, 2)])
@pytest.mark.parametrize("off_in,off_out", [(0, 0), (0, 1), (1, 1)])
def test_many_randomisations(r, r_x, n, d, off_in, off_out):
    """On both sides of the limits on a randomisation's words, and more randomisations than a grid has rows."""
    test_runs(r, r_x, n, d, off_in, off_out)


@pytest.mark.parametrize("mmax", [1, 2, 3, 5, 7, 8, 9, 17, 33, 64])
@pytest.mark.parametrize("d", [1, 3, 8, 63, 64, 65])
def test_tables(mmax, d):
    rng = np.random.Generator(np.random.SFC64(mmax * 100 + d))
    r, n = 2, min(1 << mmax, 3000)
    C, sh = rng.integers(0, 1 << 63, (r, d, mmax), dtype=U), rng.integers(0, 1 << 63, (r, d), dtype=U)
    ls = np.array([1, 0], dtype=U)
    xb, want = np.empty((r, n, d), U), np.empty((r, n, d), U)
    oracle.call("dnb2_gen_gray", U(r), U(n), U(d), U(0), U(mmax), C, xb)
    oracle.call("dnb2_digital_shift", U(r), U(n), U(d), U(r), ls, xb, sh, want)
    got = np.zeros((r, n, d), U)
    batch.dnb2_gen_fused(r, n, d, 0, mmax, C, order="gray", lshifts=ls, shiftsb=sh, xrb=got)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("alpha,bits,bits_a,mmax,lms", [(1, 64, 64, 20, True), (2, 64, 64, 17, True), (2, 31, 62, 33, True),
                                                       (3, 33, 64, 40, True), (5, 12, 60, 64, True), (4, 16, 64, 5, False),
                                                       (2, 32, 50, 1, True)])
def test_plan_matrices(alpha, bits, bits_a, mmax, lms):
    rng = np.random.Generator(np.random.SFC64(alpha * 1000 + bits))
    r, d, n = 3, 3, min(1 << mmax, 500)
    C = rng.integers(0, 1 << 63, (1, d * alpha, mmax), dtype=U) >> U(64 - bits)
    S = rng.integers(0, 1 << 63, (r, d * alpha, bits), dtype=U) * U(2) >> U(64 - bits)
    src = np.empty((r, d * alpha, mmax), U)
    if lms:
        oracle.call("dnb2_linear_matrix_scramble", U(r), U(d * alpha), U(mmax), U(1), U(bits), S, C, src)
    else:
        src[:] = C
    mat = src
    if alpha > 1:
        mat = np.empty((r, d, mmax), U)
        oracle.call("dnb2_interlace", U(r), U(d), U(mmax), U(d * alpha), U(bits), U(bits_a), U(alpha), src, mat)
    want = np.empty((r, n, d), U)
    oracle.call("dnb2_gen_gray", U(r), U(n), U(d), U(0), U(mmax), mat, want)
    xb = _cuda(np.zeros((r, n, d), U))
    req = dict(r=r, n=n, d=d, mmax=mmax, d_pre=d * alpha, alpha=alpha, tmax=bits, tmax_new=bits, tmax_alpha=bits_a,
               r_C=1, order="gray", C=_cuda(C), xb=xb)
    if lms:
        req["S"] = _cuda(S)
    batch.NetPlan([req]).run()
    assert np.array_equal(_bits(xb), want.reshape(-1))
