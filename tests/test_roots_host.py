"""Roots of unity of the FP64 digit-slice transforms (csrc/roots.hpp), on the host: every fixed-point entry within
one unit of the root, and the sums over the subgroups of order 2, 3 and 5 exactly zero (a constant line then gives
exact zeros beside its mean), for every box axis that the transforms take."""

from __future__ import annotations

import ctypes as C
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
BITS = 54
SMOOTH = [n for n in range(1, 301) if all(p in (2, 3, 5) for p in
                                          [q for q in range(2, n + 1) if n % q == 0 and all(q % d for d in range(2, q))])]


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    so = tmp_path_factory.mktemp("roots") / "libroots.so"
    cmd = ["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", str(ROOT / "ad-dft_gb300" / "csrc"),
           str(ROOT / "tests" / "c" / "roots.cpp"), "-o", str(so)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    return C.CDLL(str(so))


def roots(lib, n, forward):
    re, im = np.zeros(n, np.int64), np.zeros(n, np.int64)
    er, ei = np.zeros(n), np.zeros(n)
    lib.roots(n, forward, BITS, *(a.ctypes.data_as(C.c_void_p) for a in (re, im, er, ei)))
    return re, im, er, ei


@pytest.mark.parametrize("forward", [0, 1])
def test_sums_over_subgroups_are_zero_and_entries_within_a_unit(lib, forward):
    for n in SMOOTH:
        re, im, er, ei = roots(lib, n, forward)
        assert np.max(np.abs(er)) < 1 and np.max(np.abs(ei)) < 1, n
        assert np.max(np.abs(re)) <= 1 << BITS and np.max(np.abs(im)) <= 1 << BITS
        assert re[0] == 1 << BITS and im[0] == 0, n
        for p in (2, 3, 5):
            if n % p == 0 and n > 1:
                i = (np.arange(n)[:, None] + np.arange(p)[None] * (n // p)) % n
                assert not re[i].sum(1).any() and not im[i].sum(1).any(), (n, p)


def test_entries_are_the_roots(lib):
    """Against sums of the recurrence in 120 binary digits of Python integers."""
    from fractions import Fraction

    def atan_inv(x, one):
        s, t, k = 0, one // x, 1
        while t:
            s += t // k if k % 4 == 1 else -(t // k)
            t //= x * x
            k += 2
        return s

    P = 140
    one = 1 << P
    pi = 4 * (4 * atan_inv(5, one) - atan_inv(239, one))
    for n in (1, 2, 3, 5, 9, 16, 27, 45, 75, 80, 125, 128, 300):
        re, im, _, _ = roots(lib, n, 0)
        for t in range(0, n, max(1, n // 37)):
            a = Fraction(2 * pi * t, n * one)
            a -= Fraction(pi, one) * 2 * round(a / (2 * Fraction(pi, one)))
            x = int(a * one)
            c, s, tc, ts, k = one, x, one, x, 1
            while tc or ts:
                tc = -(((tc * x) >> P) * x >> P) // ((2 * k - 1) * (2 * k))
                ts = -(((ts * x) >> P) * x >> P) // ((2 * k) * (2 * k + 1))
                if abs(tc) <= 1 and abs(ts) <= 1:
                    break
                c, s, k = c + tc, s + ts, k + 1
            assert abs(Fraction(c, one) * (1 << BITS) - int(re[t])) < 1, (n, t)
            assert abs(Fraction(s, one) * (1 << BITS) - int(im[t])) < 1, (n, t)
