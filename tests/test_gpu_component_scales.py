"""FP64 and double-float block MVPs with components of very different size: each
keeps its own precision where components do not couple (the normal one of a
flat box, the transverse and axial ones of a chain) or couple weakly (electric
and magnetic ones at small k d), per component against the FP64 oracle.

Bound: five transforms of at most 4 x 2^-53 each (2.2e-15 of a component's norm),
the oracle's own FP64 transforms (about 1e-15) and the products; double-float
inputs are rounded before both sides see them, the result to 2^-48.
"""
import numpy as np
import pytest

import bdda
from oracle import mbt
from test_fixed_point_fft import _mvp

pytestmark = pytest.mark.gpu

TOL = 2e-14


def _check(n, f, k, x, frac, groups):
    """Relative error of each group of components, FP64 and double-float."""
    N = int(np.prod(n))
    rng = np.random.default_rng(7)
    addr = np.sort(rng.choice(N, size=max(2, int(N * frac)), replace=False)).astype(np.int32)
    x = x(rng, addr.size).reshape(f * addr.size, 2)
    hi = x.real.astype(np.float32), x.imag.astype(np.float32)      # exact in double-float
    x = (hi[0] + (x.real - hi[0]).astype(np.float32).astype(float)) + 1j * (hi[1] + (x.imag - hi[1]).astype(np.float32).astype(float))
    lf = 0.3
    gh, P = mbt.green_hat(n, f, lf, k)
    want = mbt.block_mvp(n, f, gh, P, addr, np.zeros(f * addr.size), x).reshape(addr.size, f, 2)
    op = bdda.Operator(n, lf, k, f=f)
    op.set_dipoles(addr)
    for prec in (bdda.PREC_FP64, bdda.PREC_DF64):
        y = _mvp(op, x, prec).reshape(addr.size, f, 2)
        for g in groups:
            w = np.linalg.norm(want[:, g])
            assert np.linalg.norm(y[:, g] - want[:, g]) <= TOL * w, (prec, g)


@pytest.mark.parametrize("small", [1e-3, 1e-9, 0.0])
@pytest.mark.parametrize("n, axis", [((40, 36, 1), 2), ((30, 1, 44), 1), ((1, 50, 41), 0), ((1, 1, 120), 2), ((75, 1, 1), 0),
                                     ((1, 64, 1), 1)])
@pytest.mark.parametrize("which", ["one", "others"])
def test_uncoupled_components(n, axis, small, which):
    s = np.where((np.arange(3) == axis) == (which == "one"), small, 1.0)
    x = lambda rng, m: (rng.standard_normal((m, 3, 2)) + 1j * rng.standard_normal((m, 3, 2))) * s[:, None]  # noqa: E731
    groups = [[axis], [c for c in range(3) if c != axis]]
    _check(n, 3, 1.3 + 0.02j, x, 0.8, groups)


@pytest.mark.parametrize("small", [1e-6, 1e-12, 0.0])
@pytest.mark.parametrize("kd", [1.0, 1e-4, 1e-7])
@pytest.mark.parametrize("which", [0, 1])
def test_electric_and_magnetic_components(kd, small, which):
    s = np.repeat([small, 1.0] if which == 0 else [1.0, small], 3)
    x = lambda rng, m: (rng.standard_normal((m, 6, 2)) + 1j * rng.standard_normal((m, 6, 2))) * s[:, None]  # noqa: E731
    _check((9, 12, 15), 6, kd / 0.3, x, 0.6, [[0, 1, 2], [3, 4, 5]])


def test_coupled_components_of_different_size():
    x = lambda rng, m: (rng.standard_normal((m, 3, 2)) + 1j * rng.standard_normal((m, 3, 2))) * np.array([1, 1e-4, 1e-8])[:, None]  # noqa: E731
    _check((14, 17, 20), 3, 1.3, x, 0.5, [[0], [1], [2]])
