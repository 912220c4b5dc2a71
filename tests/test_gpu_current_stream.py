"""Calls on the current stream, which enter no stream context, against the same calls on another stream:
the same results, ordered on the stream that was asked for, and the current stream left as it was."""
import numpy as np
import pytest
import torch

import qmctoolscl_gb300 as q
from qmctoolscl_gb300 import batch, tc_fft

pytestmark = pytest.mark.gpu
U = np.uint64


def _streams(which):
    """(stream argument, stream to make current, stream that the work is on)"""
    side = torch.cuda.Stream()
    return {"none": (None, None, torch.cuda.current_stream()), "none in a context": (None, side, side),
            "current": (side, side, side), "other": (side, None, side),
            "other than the context's": (side, torch.cuda.Stream(), side)}[which]


@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("which", ["none", "none in a context", "current", "other", "other than the context's"])
def test_streams(which, host):
    rng = np.random.default_rng(5)
    r, n, d, m = 2, 257, 3, 9
    C = rng.integers(0, 1 << 62, (r, d, m), dtype=U)
    sh = rng.integers(0, 1 << 62, (r, d), dtype=U)
    ls, tm = np.zeros(r, U), np.full(r, 62, U)
    x = rng.standard_normal((4, 512))
    want_b, want_x, want_h = np.empty((r, n, d), U), np.empty((r, n, d)), x.copy()
    q.dnb2_gen_gray(U(r), U(n), U(d), U(0), U(m), C, want_b)
    batch.dnb2_gen_fused(r, n, d, 0, m, C, order="gray", lshifts=ls, shiftsb=sh, tmaxes=tm, x=want_x)
    q.fwht_1d_radix2(U(4), U(1), U(256), want_h)

    stream, ctx, on = _streams(which)
    put = (lambda a: a.copy()) if host else (lambda a: torch.from_numpy(a.view(np.int64) if a.dtype == U else a).cuda())
    aC, ash, als, atm = put(C), put(sh), put(ls), put(tm)
    b, f, h, t = put(np.zeros((r, n, d), U)), put(np.zeros((r, n, d))), put(x), put(x)
    torch.cuda.synchronize()
    before = torch.cuda.current_stream()
    with torch.cuda.stream(ctx):
        current = torch.cuda.current_stream()
        q.dnb2_gen_gray(U(r), U(n), U(d), U(0), U(m), aC, b, wait=False, stream=stream)
        A = batch.dnb2_gen_fused(r, n, d, 0, m, aC, order="gray", lshifts=als, shiftsb=ash, tmaxes=atm, x=f,
                                 stream=stream)
        q.fwht_1d_radix2(U(4), U(1), U(256), h, wait=False, stream=stream.cuda_stream if stream else None)
        tc_fft.fwht_1d_tc(4, 1, 256, t, stream=stream)
        assert torch.cuda.current_stream() == current
        assert A.stream == on and A.handle == on.cuda_stream
    assert torch.cuda.current_stream() == before
    on.synchronize()
    get = (lambda a: a) if host else (lambda a: a.cpu().numpy())
    assert (get(b).view(U) == want_b).all()
    assert (get(f) == want_x).all()
    assert (get(h) == want_h).all()
    ref = x.copy()
    tc_fft.fwht_1d_tc(4, 1, 256, ref)
    assert (get(t) == ref).all()
