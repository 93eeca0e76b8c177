"""Arithmetic of the fixed-point block MVPs (fx_fft.cuh) on the host, against exact integers."""
import ctypes as ct
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def fx(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fx") / "fx_arith.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I", os.path.join(ROOT, "block-dda_gb300", "csrc"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "fx_arith.cpp"), "-o", so], check=True)
    return ct.CDLL(so)


def _ll(v):
    return np.ascontiguousarray(v, dtype=np.int64).ctypes.data_as(ct.POINTER(ct.c_longlong))


# A product drops the two low x low terms of each part (below 2^31 2^31 / 2^62 = 1 unit each) and a sum is rounded once.
@pytest.mark.parametrize("low", [0x80000000, 0x7FFFFFFF, 0x80000001, 0, 0xFFFFFFFF])
@pytest.mark.parametrize("sub", [0, 1])
def test_products_at_the_ends_of_the_low_half(fx, low, sub):
    rng = np.random.default_rng(low % 1000 + sub)
    for part in range(4):                      # which of g.re, g.im, z.re, z.im has the low word
        for _ in range(50):
            v = [int(a) for a in rng.integers(-2 ** 59, 2 ** 59, 8)]
            v[part] = (v[part] >> 32 << 32) | low
            g, z = v[0:2] + v[4:6], v[2:4] + v[6:8]
            s = [sub, 0]
            out = np.zeros(2, np.int64)
            fx.fx_products(2, _ll(g), _ll(z), np.array(s, np.int32).ctypes.data_as(ct.POINTER(ct.c_int)), 0, _ll(out))
            re = im = 0
            for i in range(2):
                sg = -1 if s[i] else 1
                a, b, c, d = g[2 * i], g[2 * i + 1], z[2 * i], z[2 * i + 1]
                re += sg * (a * c - b * d)
                im += sg * (a * d + b * c)
            assert abs(int(out[0]) * 2 ** 62 - re) <= 5 * 2 ** 62
            assert abs(int(out[1]) * 2 ** 62 - im) <= 5 * 2 ** 62


# The largest terms of a row: 3 (f = 6: and 2 in a sum of their own) with |re| + |im| <= 2^61 and |z| <= 2^61; no sum may
# wrap.
@pytest.mark.parametrize("terms, minus", [(3, 0), (5, 0), (5, 1)])
def test_largest_rows_do_not_wrap(fx, terms, minus):
    gbits = zbits = 61
    rng = np.random.default_rng(terms)
    for _ in range(400):
        g, z, s = [], [], []
        for _ in range(terms):
            a = int(rng.integers(0, 2 ** gbits)) if rng.random() < 0.5 else int(rng.choice([0, 2 ** gbits - 1, 2 ** (gbits - 1)]))
            g += [a, 2 ** gbits - 1 - a]
            z += [int(2 ** zbits * 0.7071)] * 2 if rng.random() < 0.7 else [2 ** zbits - 1, 0]
            s.append(int(rng.integers(0, 2)))
        for v in (g, z):      # low halves at both ends, signs at random
            for i in range(len(v)):
                v[i] = ((v[i] >> 32 << 32) | int(rng.choice([0x7FFFFFFF, 0x80000001, v[i] & 0xFFFFFFFF]))) * int(rng.choice([-1, 1]))
        out = np.zeros(2, np.int64)
        fx.fx_products(terms, _ll(g), _ll(z), np.array(s, np.int32).ctypes.data_as(ct.POINTER(ct.c_int)), minus, _ll(out))
        sg = [(-1 if s[i] else 1) * (-1 if minus and i > 2 else 1) for i in range(terms)]
        re = sum(sg[i] * (g[2 * i] * z[2 * i] - g[2 * i + 1] * z[2 * i + 1]) for i in range(terms))
        im = sum(sg[i] * (g[2 * i] * z[2 * i + 1] + g[2 * i + 1] * z[2 * i]) for i in range(terms))
        assert abs(int(out[0]) * 2 ** 62 - re) <= (2 * terms + 1) * 2 ** 62
        assert abs(int(out[1]) * 2 ** 62 - im) <= (2 * terms + 1) * 2 ** 62


# Elements are shifted right by e + s - ex: e the largest exponent of their line, ex their own, s from 1 to 64.
def test_shifts_of_marked_lines_stay_in_range(fx):
    fx.fx_align.restype = ct.c_longlong
    zero, bad = fx.fx_zero_exp(), fx.fx_bad_exp()
    for exps in ([bad, zero, 900, -1100], [bad, bad], [zero, 900], [-1100, zero], [bad, -1100]):
        e = max(exps)
        for ex in exps:
            assert e - ex >= 0 and -2 ** 31 <= e - ex
            for s in (1, 64):
                assert 1 <= e + s - ex < 2 ** 31 and e + s < 2 ** 31
                r = e + s - ex
                v = 2 ** 61 - 12345
                assert fx.fx_align(ct.c_longlong(v), r) == (v + 2 ** (min(r, 62) - 1)) >> min(r, 62)
    assert zero < -5000 and bad > 5000            # beyond every exponent of a value
