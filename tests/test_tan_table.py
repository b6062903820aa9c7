"""The native FP64 register passes' twiddle tables (CPU): every entry of every stage against twiddles in longer arithmetic.

A twiddle is w_q = i^m c_q (1 + i t_q), the t rounded once and the scale c made for the rounded t; the table holds the t,
ratios of scales, and two bits of m a value.  The oracle tests' tolerances would not see a wrong last bit or an entry of
a rare j."""
import ctypes

import numpy as np
import pytest

from decomp_mpi_gb300._lib import load

U = np.longdouble(2) ** -53
LENGTHS = [32, 48, 64, 96, 120, 128, 160, 192, 240, 256, 320, 384, 480, 512, 1024]


def _tables(n, reg, sign):
    """(radix, points before it, entries [e, j] as pairs of doubles) of the stages after the first."""
    lib = load()
    lib.dmg_fft_tan_entries.argtypes = [ctypes.c_int] * 3 + [ctypes.POINTER(ctypes.c_double)]
    lib.dmg_fft_reg_radices.argtypes = [ctypes.c_int] * 4 + [ctypes.POINTER(ctypes.c_int)] * 2
    first, last = ctypes.c_int(), ctypes.c_int()
    lib.dmg_fft_reg_radices(0, n, reg, sign, ctypes.byref(first), ctypes.byref(last))
    middle = n // (first.value * last.value)
    stages = ([middle] if middle > 1 else []) + [last.value]
    count = lib.dmg_fft_tan_entries(n, reg, sign, None)
    buf = (ctypes.c_double * (2 * count))()
    assert lib.dmg_fft_tan_entries(n, reg, sign, buf) == count
    flat = np.array(buf[:]).reshape(count, 2)
    out, at, lp = [], 0, first.value
    for r in stages:
        out.append((r, lp, flat[at:at + r * lp].reshape(r, lp, 2)))
        at += r * lp
        lp *= r
    assert at == count and lp == n
    return out


@pytest.mark.skipif(np.finfo(np.longdouble).eps > 2.0 ** -60, reason="no longer float on the host")
@pytest.mark.parametrize("sign", [-1, 1])
@pytest.mark.parametrize("reg", [1, 2], ids=["v1", "t"])
@pytest.mark.parametrize("n", LENGTHS)
def test_entries(n, reg, sign):
    pi = np.longdouble("3.141592653589793238462643383279502884")
    for r, lp, e in _tables(n, reg, sign):
        assert r in (4, 8)
        v = e.transpose(1, 0, 2).reshape(lp, 2 * r)  # a row per j
        t = v[:, :r - 1].astype(np.longdouble)
        if r == 8:
            rho, (c2, c31, c1, c1h), word = v[:, 7:11], v[:, 11:15].T, v[:, 15]
            scale = [None, c1, c2, c31 * np.longdouble(1) * c1]
            scale += [rho[:, q] * (np.longdouble(1) if q == 0 else np.longdouble(1) * scale[q]) for q in range(4)]
            # the eighth turn's scale, rounded once from c_1's unrounded value
            assert np.all(np.abs(c1h - scale[1] * np.sqrt(np.longdouble(0.5))) <= 2 * U)
        else:
            c2, c31, c1 = v[:, 3], v[:, 4], v[:, 5]
            word = v[:, 6]
            scale = [None, c1, c2, c31 * np.longdouble(1) * c1]
        code = np.ascontiguousarray(word).view(np.uint64)
        j = np.arange(lp)
        for q in range(1, r):
            tq, c = t[:, q - 1], scale[q]
            assert np.all(np.abs(tq) <= 1)
            # one rounding of the scale of the rounded t, made for the rounded scales below it
            exact = 1 / np.sqrt(1 + tq * tq)
            assert np.all(np.abs(c - exact) <= 1.01 * U * exact), (n, r, q)
            m = ((code >> np.uint64(2 * (q - 1))) & np.uint64(3)).astype(int)
            re, im = c, c * tq
            for turn in range(1, 4):
                pick = m >= turn
                re, im = np.where(pick, -im, re), np.where(pick, re, im)
            a = sign * 2 * pi * (q * j).astype(np.longdouble) / (r * lp)
            # t to half a unit below 1 (2^-54) and the scale to one: 2 U covers both parts
            assert np.all(np.abs(re - np.cos(a)) <= 2 * U) and np.all(np.abs(im - np.sin(a)) <= 2 * U), (n, r, q)
