"""The straight-line reciprocal, quotient and square root of the stage kernels
against the correctly rounded operators, bit for bit: random operands over the
stated range, significands near 1 and 2 and of all ones, the ends of the range
and zero, and the hard cases, whose exact result lies next to the middle of two
neighbours -- there alone can the last correction go to the wrong side."""
import ctypes

import numpy as np
import pytest

from ptha_b200 import _lib

pytestmark = pytest.mark.gpu

RECIPROCAL, QUOTIENT, ROOT = 0, 1, 2


def _rounded(op, a, b=None):
    a = np.ascontiguousarray(a, dtype=np.float64)
    b = None if b is None else np.ascontiguousarray(b, dtype=np.float64)
    out = np.empty_like(a)
    p = [None if x is None else x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, out)]
    _lib.check(_lib.lib().swals_gpu_rounded(op, p[0], p[1], a.size, p[2]))
    return out


def _same(got, want):
    bad = np.flatnonzero(got.view(np.int64) != want.view(np.int64))
    assert bad.size == 0, (bad.size, bad[:5], got[bad[:5]], want[bad[:5]])


def _operands(rng, n, emin, emax):
    """Significands random, within 2^-44 of 1 and of 2, with 29 leading ones."""
    m = rng.integers(0, 1 << 52, n, dtype=np.int64)
    kind = rng.integers(0, 8, n)
    m = np.where(kind == 4, m | 0xFFFFFFFFFFF00, m)
    m = np.where(kind == 5, m & 0xFF, m)
    m = np.where(kind == 6, m | 0xFFFFFFF000000, m)
    m = np.where(kind == 7, (1 << 52) - 1, m)
    e = rng.integers(emin, emax + 1, n, dtype=np.int64) + 1023
    return ((e << 52) | m).view(np.float64)


N = 1 << 21


def test_random_operands():
    rng = np.random.default_rng(7)
    b = _operands(rng, N, -963, 962) * rng.choice([-1.0, 1.0], N)
    _same(_rounded(RECIPROCAL, b), 1.0 / b)
    a, b = _operands(rng, N, -481, 480) * rng.choice([-1.0, 1.0], N), _operands(rng, N, -481, 480)
    _same(_rounded(QUOTIENT, a, b), a / b)
    x = _operands(rng, N, -963, 1023)
    _same(_rounded(ROOT, x), np.sqrt(x))
    assert np.isnan(_rounded(ROOT, np.array([np.inf, np.nan]))).all()


def test_ends_of_the_range():
    ends = np.array([1.0e-290, np.nextafter(1.0e-290, 1), 1.0e-5, 1.0, 1.0e30, 1.0e280, np.nextafter(1.0e290, 0)])
    _same(_rounded(RECIPROCAL, ends), 1.0 / ends)
    a, b = (x.ravel() for x in np.meshgrid(ends, ends))
    with np.errstate(over="ignore", under="ignore"):
        ok = (a / b >= 1.0e-290) & (a / b <= 1.0e290)
    _same(_rounded(QUOTIENT, a[ok], b[ok]), a[ok] / b[ok])
    _same(_rounded(ROOT, ends), np.sqrt(ends))
    below = np.array([0.0, 5.0e-324, 2.3e-308, np.nextafter(1.0e-290, 0)])
    _same(_rounded(ROOT, below), np.zeros(4))


def test_reciprocals_next_to_a_middle():
    # (2^53 - k) (2^53 + k) = 2^106 - k^2: 1/(2^53 - k) is just above the middle
    # (2^53 + k) / 2^106 for odd k
    k = np.arange(0, 1 << 20)
    b = (float(1 << 53) - k) * 2.0 ** -53
    _same(_rounded(RECIPROCAL, b), 1.0 / b)
    b = 1.0 + k * 2.0 ** -52
    _same(_rounded(RECIPROCAL, b), 1.0 / b)


def _hard_quotients(B, offsets):
    """(A, B) of 53 bits with A 2^s = B M + c, M / 2^54 or M / 2^53 the middle
    of two quotients."""
    out = []
    for b in B:
        inv = pow(b, -1, 1 << 54)
        for c in offsets:
            for s in (54, 53):
                M = (-c * inv) % (1 << s)
                if s == 53:
                    M += 1 << 53
                A = (b * M + c) >> s
                if M % 2 and M > 1 << 53 and 1 << 52 <= A < 1 << 53:
                    out.append((A, b))
    return out


def test_quotients_next_to_a_middle():
    rng = np.random.default_rng(11)
    # divisors near 2, whose reciprocals are next to a middle themselves, and any
    near = [(1 << 53) - k for k in range(1, 1 << 15, 2)]
    any_ = [int(b) | 1 for b in rng.integers(1 << 52, 1 << 53, 20000)]
    pairs = _hard_quotients(near, (-1, 1, -3, 3)) + _hard_quotients(any_, (-1, 1))
    assert len(pairs) > 40000
    a, b = np.array(pairs, dtype=np.int64).T.astype(np.float64)
    for ea, eb in ((0, 0), (-52, -52), (-40, 400), (300, -100)):
        x, y = np.ldexp(a, ea), np.ldexp(b, eb)
        _same(_rounded(QUOTIENT, x, y), x / y)


def _hard_roots(limit):
    """X with X 2^54 = M^2 - s, |s| <= limit: sqrt(X / 2^52) next to the middle
    M / 2^53 of two roots.  M^2 = s mod 2^54 (s = 1 mod 8) by lifting roots bit
    by bit."""
    out = []
    for s in range(-limit, limit + 1):
        if s % 8 != 1:
            continue
        roots = [r for r in range(8) if (r * r - s) % 8 == 0]
        for k in range(4, 55):
            roots = sorted({r + t for r in roots for t in (0, 1 << (k - 1), 1 << (k - 2))
                            if ((r + t) ** 2 - s) % (1 << k) == 0 and r + t < 1 << k})
        for M in roots:
            X = (M * M - s) >> 54
            if M > 1 << 53 and (X < 1 << 53 or X % 2 == 0) and X >= 1 << 52:
                out.append(X)
    return out


def test_roots_next_to_a_middle():
    X = _hard_roots(1000)
    assert len(X) > 250
    x = np.array(X, dtype=np.int64).astype(np.float64)
    assert all(int(v) == q for v, q in zip(x, X))
    for e in (-52, -1012, -512, 0, 500, 900, 970):
        y = np.ldexp(x, e)
        _same(_rounded(ROOT, y), np.sqrt(y))
