"""The DFT constants of the register transforms (cubokit_b200/csrc/regdft.cuh) are cos and sin of 2 pi k / R rounded to the
nearest double, every radix and k.  They reach every FP64 pass: constants a unit off act as one gain on all positions."""
import ctypes as C
import subprocess
from decimal import Decimal, getcontext
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
SRC = ROOT / "tests" / "cuda" / "turns_probe.cu"
getcontext().prec = 60
PI = Decimal("3.14159265358979323846264338327950288419716939937510582097494459230781640628620899")


@pytest.fixture(scope="module")
def turns(tmp_path_factory):
    from cubokit_b200.build import nvcc
    lib = tmp_path_factory.mktemp("turns") / "libturns_probe.so"
    subprocess.run([nvcc(), "-std=c++17", "--expt-relaxed-constexpr", "-gencode", "arch=compute_100a,code=sm_100a", "-shared",
                    "-Xcompiler", "-fPIC", "-I", str(ROOT / "cubokit_b200" / "csrc"), str(SRC), "-o", str(lib)], check=True)
    return C.CDLL(str(lib)).turns


def _series(x, first):
    term = x if first else Decimal(1)
    total = term
    for i in range(1, 60):
        term = -term * x * x / ((2 * i - 1 + first) * (2 * i + first))
        total += term
    return total


def _rounded(k, n):
    """cos and sin of 2 pi k / n: the exact ones on the axes, else their series, rounded once."""
    if 4 * k % n == 0:
        return [(1, 0), (0, 1), (-1, 0), (0, -1)][4 * k // n % 4]
    x = 2 * PI * k / n
    return float(_series(x, 0)), float(_series(x, 1))


@pytest.mark.parametrize("radix", range(2, 32))
def test_every_constant_is_the_nearest_double(turns, radix):
    c, s = np.empty(radix), np.empty(radix)
    p = C.POINTER(C.c_double)
    assert turns(radix, c.ctypes.data_as(p), s.ctypes.data_as(p)) == 0
    want = np.array([_rounded(k, radix) for k in range(radix)], np.float64)
    assert np.array_equal(c, want[:, 0]) and np.array_equal(s, want[:, 1])
