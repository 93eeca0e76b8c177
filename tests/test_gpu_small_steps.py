"""Gram sums and one-CTA L x L steps of the solvers at the block widths where
their split changes: one column, the widest block whose Gram rows are split
over threads (8) and the next, a full tile of 16 and the next, and 32."""
import numpy as np
import pytest

import bdda
from oracle import mbt

pytestmark = pytest.mark.gpu

TRUE_TOL = 1e-8


# The solve stops on true residuals from the device's matvec, whose rounding (1e-15 of |x| |A|, far below 1e-3 of the
# tolerance) is all that separates them from the oracle's.
@pytest.mark.parametrize("L", [1, 8, 9, 16, 17, 32])
@pytest.mark.parametrize("solver, precision", [("cocg_rq", bdda.SOLVE_FP64), ("cocg_rq", bdda.SOLVE_MIXED),
                                               ("bicgstab", bdda.SOLVE_FP64), ("bicggr", bdda.SOLVE_FP64)])
def test_block_widths(solver, precision, L):
    prob = bdda.make_problem(150, 1.7 + 0.3j, seed=21, n_dirs=(L + 1) // 2)
    B = np.asfortranarray(prob.B[:, :L])
    op = bdda.Operator(prob.n, prob.lf, prob.k)
    op.set_dipoles(prob.address)
    X, st = bdda.solve(op, prob.diag, B, bdda.solve_opts(solver, jacobi=True, precision=precision, tol=1e-8,
                                                         true_tol=TRUE_TOL, itermax=600))
    assert st["status"] == 0
    gh, P = mbt.green_hat(prob.n, 3, prob.lf, prob.k)
    R = B - mbt.block_mvp(prob.n, 3, gh, P, prob.address, prob.diag, X)
    assert np.all(np.linalg.norm(R, axis=0) <= TRUE_TOL * 1.001 * np.linalg.norm(B, axis=0))
