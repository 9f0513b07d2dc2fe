"""The folded transforms' tables and index algebra (csrc/dft.cu) on the CPU: the sums
that the kernels form from a table, with the folding of the input, the second folding
of even lengths and the mirrored outputs, against numpy's FFT, for every length up to
130 and some up to the last that can be served, with the tables of both axes and
precisions (different tiles).  FP64 arithmetic; a sum of K <= 513 products of values
below 1 has an error below 513 * 2**-52, asked for here as 1e-12.
"""
import ctypes

import numpy as np
import pytest

from conftest import ehd

STAGE = 16


def fn(symbol, res, args):
    f = getattr(ehd.lib(), symbol)
    f.restype, f.argtypes = res, args
    return f


def table(n, y, rsize):
    sz, b, i = ctypes.c_size_t, ctypes.c_bool, ctypes.c_int
    pitch = fn("_ZN3ehd15dft_table_pitchEibm", i, [i, b, sz])(n, y, rsize)
    elems = fn("_ZN3ehd15dft_table_elemsEibm", sz, [i, b, sz])(n, y, rsize)
    t = np.empty(2 * elems)
    fn("_ZN3ehd9dft_tableEibmPd", None, [i, b, sz, ctypes.POINTER(ctypes.c_double)])(
        n, y, rsize, t.ctypes.data_as(ctypes.POINTER(ctypes.c_double)))
    return t.reshape(-1, pitch, 2)


def transform(v, t):
    """sum_a v_a exp(-2 pi i a b / n), b = 0..n-1, of the columns of a complex v as the
    y kernels form it."""
    n, h = len(v), len(v) // 2
    even = n % 2 == 0
    stages = lambda m: (m + STAGE - 1) // STAGE
    te = stages(h // 2 + 1) if even else stages(h + 1)
    rows = np.arange(t.shape[0])
    a = np.where(rows < STAGE * te, 2 * rows, 2 * (rows - STAGE * te) + 1) if even else rows
    s, d = np.zeros((len(a),) + v.shape[1:], complex), np.zeros((len(a),) + v.shape[1:], complex)
    for r, x in enumerate(a):
        if 2 * x > n:
            continue
        pair = x > 0 and 2 * x < n
        s[r] = v[x] + (v[n - x] if pair else 0)
        d[r] = v[x] - v[n - x] if pair else 0
    cos = lambda part: np.tensordot(t[part, :, 0].T, s[part], 1)
    sin = lambda part: np.tensordot(t[part, :, 1].T, d[part], 1)
    out = np.full(v.shape, np.nan, complex)

    def emit(b, c, w):
        out[b] = c - 1j * w
        if b > 0 and 2 * b < n:
            out[n - b] = c + 1j * w

    if not even:
        c, w = cos(slice(None)), sin(slice(None))
        for b in range(h + 1):
            emit(b, c[b], w[b])
        return out
    lo, hi = slice(0, STAGE * te), slice(STAGE * te, None)
    ce, se, co, so = cos(lo), sin(lo), cos(hi), sin(hi)
    for b in range(h // 2 + 1):
        if 2 * b <= h:
            emit(b, ce[b] + co[b], se[b] + so[b])
        if 2 * b < h:
            emit(h - b, ce[b] - co[b], so[b] - se[b])
    return out


@pytest.mark.parametrize("rsize", [4, 8])
@pytest.mark.parametrize("y", [False, True])
def test_folded_sums_are_the_dft(y, rsize):
    rng = np.random.default_rng(1)
    for n in list(range(1, 131)) + [183, 251, 360, 386, 509, 768, 1021, 1022, 1023, 1024]:
        v = rng.uniform(-1, 1, (n, 3)) + 1j * rng.uniform(-1, 1, (n, 3))
        got = transform(v, table(n, y, rsize))
        assert np.abs(got - np.fft.fft(v, axis=0)).max() < 1e-12 * max(1, n / 16), n
