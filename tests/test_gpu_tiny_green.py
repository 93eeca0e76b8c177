"""Green tensors below 2^-923 (strong absorption between neighbouring sites):
the spectrum's transforms scale such lines up before they convert them, and it
is packed with all its bits."""
import numpy as np
import pytest

import bdda
from oracle import mbt
from test_fixed_point_fft import _mvp, _rel

pytestmark = pytest.mark.gpu


# exp(-k_im lf) = 2^-bits at one site's distance, and G is |k|^2 / lf = 2^25 times that
@pytest.mark.parametrize("bits", [958, 985, 1010])
@pytest.mark.parametrize("n", [(5, 6, 7), (33, 20, 40), (2, 65, 64)])
def test_strong_absorption(n, bits):
    lf = 0.25
    k = 1.0 + 1j * (bits * np.log(2) / lf)
    rng = np.random.default_rng(bits)
    N = int(np.prod(n))
    addr = np.sort(rng.choice(N, size=N // 2, replace=False)).astype(np.int32)
    x = rng.standard_normal((3 * addr.size, 2)) + 1j * rng.standard_normal((3 * addr.size, 2))
    gh, P = mbt.green_hat(n, 3, lf, k)
    want = mbt.block_mvp(n, 3, gh, P, addr, np.zeros(3 * addr.size), x)
    op = bdda.Operator(n, lf, k)
    op.set_dipoles(addr)
    assert 0 < np.abs(gh).max() < 2.0 ** -923
    assert _rel(_mvp(op, x, bdda.PREC_FP64) * 2.0 ** 900, want * 2.0 ** 900) <= 1e-12   # the suite's bar for FP64 MVPs
