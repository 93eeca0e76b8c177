"""The z pass of complex FP32 for lines below 181 points (a CTA shares out the
butterflies of several (line, right-hand side) tasks), at the ends of its range
and at odd right-hand-side counts, against the FP64 block MVP."""
import numpy as np
import pytest

import bdda

pytestmark = pytest.mark.gpu

# FP32 transforms of three axes: the bound the other plan tests use
TOL32 = 5e-6


# z lengths 6 = 2 3 (the shortest two-stage line), 8, 32, 90, 125 = 5 5 5 (three stages), 128 = 16 8, 150 = 15 10
# (not the operator's 10 15), 162 (three stages, not in range) and 180 (the longest)
@pytest.mark.parametrize("nz", [3, 4, 16, 45, 62, 64, 75, 81, 90])
@pytest.mark.parametrize("L", [1, 2, 7])
def test_short_z_lines(nz, L):
    import torch
    n = (3, 5, nz)  # 6 x 10 lines: the last CTA of two to four tasks is partly empty at odd task counts
    rng = np.random.default_rng(100 * nz + L)
    N = int(np.prod(n))
    addr = np.sort(rng.choice(N, size=(2 * N) // 3, replace=False)).astype(np.int32)
    rows = 3 * addr.size
    x = rng.standard_normal((L, rows)) + 1j * rng.standard_normal((L, rows))
    op = bdda.Operator(n, 0.03, 2 * np.pi / 0.55)
    op.set_dipoles(addr)

    def mvp(prec, dt):
        xd = torch.from_numpy(x).to(dt).cuda()
        yd = torch.zeros_like(xd)
        torch.cuda.synchronize()
        op.mvp_device(xd.data_ptr(), yd.data_ptr(), L, rows, rows, prec=prec)
        torch.cuda.synchronize()
        return yd.cpu().numpy().astype(np.complex128)

    y64 = mvp(bdda.PREC_FP64, torch.complex128)
    for kind in ("default", "scalar", "packed"):
        op.set_z_kernel(kind)
        y = mvp(bdda.PREC_FP32, torch.complex64)
        assert np.linalg.norm(y - y64) <= TOL32 * np.linalg.norm(y64), kind
