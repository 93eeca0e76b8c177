"""Block MVPs of different precisions of one operator in flight on two streams:
each precision has a workspace of its own, so neither order nor a growing
buffer of the other one shows in the results."""
import numpy as np
import pytest

import bdda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first, second", [(bdda.PREC_FP64, bdda.PREC_DF64), (bdda.PREC_DF64, bdda.PREC_FP64),
                                           (bdda.PREC_FP32, bdda.PREC_DF64)])
def test_two_precisions_on_two_streams(first, second):
    import torch
    nocc, L = 4000, (4, 8)
    n, addr = bdda.aggregate(nocc, 1.0, 2.6, 5)
    rows = 3 * nocc
    rng = np.random.default_rng(11)
    dt = {bdda.PREC_FP64: torch.complex128, bdda.PREC_FP32: torch.complex64}
    xs = []
    for prec, ncol in zip((first, second), L):
        x = torch.from_numpy(rng.standard_normal((ncol, rows)) + 1j * rng.standard_normal((ncol, rows)))
        if prec == bdda.PREC_DF64:
            v = torch.view_as_real(x)
            hi = v.float()
            x = torch.stack([hi, (v - hi.double()).float()], -1).flatten(-2).contiguous()   # re_hi re_lo im_hi im_lo
        else:
            x = x.to(dt[prec])
        xs.append(x.cuda())

    def operator():
        op = bdda.Operator(n, 0.02, 2 * np.pi / 0.55)
        op.set_dipoles(addr)
        return op

    def call(op, i, y, st):
        op.mvp_device(xs[i].data_ptr(), y.data_ptr(), L[i], rows, rows, prec=(first, second)[i], stream=st.cuda_stream)

    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    op = operator()
    want = []
    for i in range(2):
        y = torch.zeros_like(xs[i])
        torch.cuda.synchronize()
        call(op, i, y, streams[i])
        torch.cuda.synchronize()
        want.append(y)
    for op in (operator(), op):     # buffers that grow while the other call runs, and buffers that are there
        got = [[torch.zeros_like(x) for _ in range(4)] for x in xs]
        torch.cuda.synchronize()
        for r in range(4):
            for i in range(2):
                call(op, i, got[i][r], streams[i])
        torch.cuda.synchronize()
        for i in range(2):
            for y in got[i]:
                assert torch.equal(y, want[i])
