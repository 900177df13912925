"""Scratch of the digit-slice products (csrc/ozlayout.hpp), on the host: every piece of a product that
goes in pieces stays within the buffer, and the pieces cover the product once."""

from __future__ import annotations

import ctypes as C
import random
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CAP = 384 << 20          # scratch that the entry points ask for at most


@pytest.fixture(scope="module")
def oz(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    so = tmp_path_factory.mktemp("oz") / "liboz.so"
    cmd = ["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I", str(ROOT / "ad-dft_gb300" / "csrc"),
           str(ROOT / "tests" / "c" / "oz_pieces.cpp"), "-o", str(so)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    lib = C.CDLL(str(so))
    lib.oz_most.restype = lib.oz_whole.restype = C.c_size_t
    lib.oz_most.argtypes = [C.c_int] * 5 + [C.c_size_t, C.POINTER(C.c_double), C.POINTER(C.c_int), C.POINTER(C.c_int)]
    return lib


def pieces(lib, digits, r, c, k, batch, nbytes):
    cov, splits, n = C.c_double(), C.c_int(), C.c_int()
    most = lib.oz_most(digits, r, c, k, batch, nbytes, C.byref(cov), C.byref(splits), C.byref(n))
    return most, cov.value, splits.value, n.value


# remainders whose own best split count needs more scratch than the whole piece's
@pytest.mark.parametrize("digits,r,c,k,nbytes", [
    (7, 591, 1316, 25984, CAP), (7, 1316, 591, 25984, CAP), (7, 485, 970, 16388, CAP), (7, 588, 801, 37020, CAP),
    (7, 282, 699, 25420, CAP), (8, 1280, 320, 2432, 70 << 20), (7, 1280, 320, 2432, 70 << 20)])
def test_remainders_stay_within_the_scratch(oz, digits, r, c, k, nbytes):
    for a, b in ((r, c), (c, r)):
        most, cov, _, n = pieces(oz, digits, a, b, k, 1, nbytes)
        assert most <= nbytes
        assert n == 0 or cov == float(a) * b * k


def test_random_products_in_random_scratch(oz):
    rng = random.Random(7)
    cut = 0
    for _ in range(20000):
        digits = rng.choice([7, 8])
        r, c, k = (int(2 ** rng.uniform(0, e)) for e in (11.5, 11.5, 15.5))
        batch = rng.choice([1, 1, 2, 3, 8, 27])
        whole = oz.oz_whole(digits, r, c, k, batch)
        nbytes = min(CAP, max(1 << 20, int(whole * rng.uniform(0.02, 1.1))))
        most, cov, _, n = pieces(oz, digits, r, c, k, batch, nbytes)
        if n == 0:
            continue
        assert most <= nbytes, (digits, r, c, k, batch, nbytes)
        assert cov == float(batch) * r * c * k
        cut += n > 1
    assert cut > 2000
