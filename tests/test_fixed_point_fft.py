"""The 64-bit fixed-point FFT core of the FP64 and double-float block MVPs.

CPU: the core on one line (the host build of the device code) against the DFT
in extended precision, for every 5-smooth length, next to the FP64 core it
replaced: dense and half-empty lines, a single nonzero, values at both ends of
FP64's range, zeros, infinities and NaN.

GPU (-m gpu): what a scale per line has to get right in a whole MVP -- columns
of very different magnitude in one call, subnormal and huge vectors, a NaN in
one right-hand side leaving the others alone -- and every axis length that
changes the plans, in FP64 and double-float.

Tolerances: the output is rounded to 53 bits (2^-54 of each part, rms), and a
transform of at most four stages adds under two units of a scale that keeps at
least 54 bits below the line's rms, so 4 x 2^-53 bounds the relative L2 error
of a dense line; a whole MVP has five such transforms and the FP64 Green
tensor, and the repository's bar for it against the oracle is 1e-12.
"""
import numpy as np
import pytest

import bdda
from oracle import mbt

EPS = 2.0 ** -53
SMOOTH = [2 ** a * 3 ** b * 5 ** c for a in range(11) for b in range(7) for c in range(5)
          if 2 <= 2 ** a * 3 ** b * 5 ** c <= 1200]


def _dft(x, inverse=False):
    """DFT in extended precision: (re, im)."""
    n = len(x)
    t = np.arange(n)
    ph = (np.outer(t, t) % n).astype(np.longdouble) * (2 * np.longdouble("3.14159265358979323846264338327950288") / n)
    c, s = np.cos(ph), np.sin(ph) * (1 if inverse else -1)
    a, b = x.real.astype(np.longdouble), x.imag.astype(np.longdouble)
    return c @ a - s @ b, s @ a + c @ b


def _order(radices, n):
    """Frequency at each output position of the forward transform."""
    q, k, w, m = np.arange(n), np.zeros(n, int), 1, n
    for r in radices:
        m //= r
        k += w * (q // m)
        q = q % m
        w *= r
    return k


def _err(y, re, im):
    return float(np.sqrt(((y.real - re) ** 2 + (y.imag - im) ** 2).sum() / (re ** 2 + im ** 2).sum()))


@pytest.mark.parametrize("n", sorted(SMOOTH))
def test_line_against_extended_precision(n):
    rng = np.random.default_rng(n)
    x = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    re, im = _dft(x)
    y, rad = bdda.host_fft_line(x, prec=4)
    assert int(np.prod(rad)) == n and max(rad) <= 10
    k = _order(rad, n)
    ours = _err(y, re[k], im[k])
    y64, rad64 = bdda.host_fft_line(x, prec=1)
    k64 = _order(rad64, n)
    assert ours <= 4 * EPS
    assert ours <= max(_err(y64, re[k64], im[k64]), EPS)   # no less precise than the FP64 transform
    # half-empty line (the MVP's padding; the hook poisons what must not be read)
    nv = max(1, n // 2)
    xp = x.copy()
    xp[nv:] = 0
    re, im = _dft(xp)
    y, _ = bdda.host_fft_line(xp, prec=4, nvalid=nv)
    assert _err(y, re[k], im[k]) <= 4 * EPS
    # inverse: digit-reversed input, the first half of the outputs
    xs = np.zeros(n, complex)
    xs[k] = x
    re, im = _dft(xs, inverse=True)
    y, _ = bdda.host_fft_line(x, inverse=True, prec=4)
    h = n // 2
    assert np.sqrt(((y[:h].real - re[:h]) ** 2 + (y[:h].imag - im[:h]) ** 2).sum()
                   / (re ** 2 + im ** 2).sum()) <= 4 * EPS


@pytest.mark.parametrize("scale", [5e-324, 3e-310, 1e-250, 1.0, 1e290])
@pytest.mark.parametrize("n", [12, 250, 1200])
def test_line_over_the_range_of_fp64(n, scale):
    rng = np.random.default_rng(n)
    m = np.round(rng.uniform(-900, 900, (n, 2)))          # exact multiples of the scale, subnormal ones too
    x = m[:, 0] * scale + 1j * (m[:, 1] * scale)
    re, im = _dft((m[:, 0] + 1j * m[:, 1]))
    y, rad = bdda.host_fft_line(x, prec=4)
    k = _order(rad, n)
    got = (y.real.astype(np.longdouble) / np.longdouble(scale)) + 1j * (y.imag.astype(np.longdouble) / np.longdouble(scale))
    quantum = 0.5 * (5e-324 / scale) if scale < 1e-300 else 0.0   # subnormal outputs are rounded to their spacing
    d = np.sqrt((np.abs(got - (re[k] + 1j * im[k])) ** 2).sum() / n)
    assert d <= 4 * EPS * np.sqrt((re ** 2 + im ** 2).sum() / n) + 2 * quantum


@pytest.mark.parametrize("n", [8, 90, 243])
def test_single_value_zeros_and_nonfinite(n):
    x = np.zeros(n, complex)
    y, _ = bdda.host_fft_line(x, prec=4)
    assert not y.any()
    x[n // 3] = 1.25 - 0.5j
    y, rad = bdda.host_fft_line(x, prec=4)
    re, im = _dft(x)
    k = _order(rad, n)
    assert _err(y, re[k], im[k]) <= 2 * EPS
    for bad in (np.nan, np.inf, -np.inf):
        x[n // 2] = complex(0, bad)
        y, _ = bdda.host_fft_line(x, prec=4)
        assert np.isnan(y.real).all() and np.isnan(y.imag).all()


# ---------------------------------------------------------------- GPU

def _to_df(a):
    hi = np.stack([a.real, a.imag], -1).astype(np.float32)
    lo = (np.stack([a.real, a.imag], -1) - hi.astype(np.float64)).astype(np.float32)
    return np.ascontiguousarray(np.stack([hi[..., 0], lo[..., 0], hi[..., 1], lo[..., 1]], -1))


def _mvp(op, x, prec, diag=None):
    """x (rows, L) complex128 -> (rows, L), through device buffers of the precision."""
    import torch
    rows, L = x.shape
    xh = np.ascontiguousarray(x.T)
    xd = torch.from_numpy(xh if prec == bdda.PREC_FP64 else _to_df(xh)).cuda()
    dd = None if diag is None else torch.from_numpy(diag if prec == bdda.PREC_FP64 else _to_df(diag)).cuda()
    yd = torch.zeros_like(xd)
    torch.cuda.synchronize()
    op.mvp_device(xd.data_ptr(), yd.data_ptr(), L, rows, rows, prec=prec, diag=dd.data_ptr() if dd is not None else None)
    torch.cuda.synchronize()
    y = yd.cpu().numpy()
    if prec != bdda.PREC_FP64:
        y = y.astype(np.float64)
        y = (y[..., 0] + y[..., 1]) + 1j * (y[..., 2] + y[..., 3])
    return y.T


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.gpu
def test_columns_of_different_magnitude_keep_their_own_scale():
    nocc, L = 260, 5
    n, addr = bdda.aggregate(nocc, 1.0, 2.4, 8)
    rng = np.random.default_rng(3)
    x = rng.standard_normal((3 * nocc, L)) + 1j * rng.standard_normal((3 * nocc, L))
    diag = rng.standard_normal(3 * nocc) + 5.0
    lf, k = 0.02, 2 * np.pi / 0.55
    gh, P = mbt.green_hat(n, 3, lf, k)
    ref = mbt.block_mvp(n, 3, gh, P, addr, diag.astype(complex), x)
    op = bdda.Operator(n, lf, k)
    op.set_dipoles(addr)
    for prec, scales in ((bdda.PREC_FP64, [1e-290, 1e-20, 1.0, 1e20, 1e280]), (bdda.PREC_DF64, [1e-20, 1e-5, 1.0, 1e5, 1e20])):
        y = _mvp(op, x * np.array(scales), prec, diag.astype(complex))
        for j, s in enumerate(scales):
            assert _rel(y[:, j] / s, ref[:, j]) <= 1e-12, (prec, s)
    # a zero column stays zero, a column with one NaN is NaN in its off-diagonal sums, the others are untouched
    xz = x.copy()
    xz[:, 1] = 0
    xz[7, 3] = np.nan
    y = _mvp(op, xz, bdda.PREC_FP64)
    clean = _mvp(op, x, bdda.PREC_FP64)
    assert not y[:, 1].any()
    assert np.isnan(y[:, 3]).all()
    for j in (0, 2, 4):
        assert np.array_equal(y[:, j], clean[:, j])


@pytest.mark.gpu
@pytest.mark.parametrize("f", [3, 6])
@pytest.mark.parametrize("n", [(1, 1, 1), (1, 2, 3), (2, 1, 9), (9, 17, 33), (5, 8, 130), (130, 3, 6), (4, 200, 7)])
def test_boxes_at_plan_and_tile_edges(n, f):
    rng = np.random.default_rng(sum(n) + f)
    N = int(np.prod(n))
    nocc = max(1, (3 * N) // 5)
    addr = np.sort(rng.choice(N, size=nocc, replace=False)).astype(np.int32)
    L = 2
    x = rng.standard_normal((f * nocc, L)) + 1j * rng.standard_normal((f * nocc, L))
    diag = rng.standard_normal(f * nocc) + 1j * rng.standard_normal(f * nocc) + 4.0
    lf, k = 0.3, 1.9 + 0.04j
    gh, P = mbt.green_hat(n, f, lf, k)
    ref = mbt.block_mvp(n, f, gh, P, addr, diag, x)
    op = bdda.Operator(n, lf, k, f=f)
    op.set_dipoles(addr)
    for prec in (bdda.PREC_FP64, bdda.PREC_DF64):
        assert _rel(_mvp(op, x, prec, diag), ref) <= 1e-12
