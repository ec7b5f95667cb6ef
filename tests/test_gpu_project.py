"""The projection's modulus and ratio from one corrected reciprocal square root (cubokit_b200/csrc/project.cuh) against
the correctly rounded square root and division, and the values that take the general functions: zeros, tiny, huge and not
finite ones, alone and beside ordinary ones."""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
SRC = ROOT / "tests" / "cuda" / "project_probe.cu"
LIB = ROOT / "tests" / "cuda" / "libproject_probe.so"


def _lib():
    csrc = ROOT / "cubokit_b200" / "csrc"
    deps = [SRC, csrc / "project.cuh", csrc / "common.cuh"]
    if not LIB.exists() or any(d.stat().st_mtime > LIB.stat().st_mtime for d in deps):
        from cubokit_b200.build import ARCH, nvcc
        subprocess.run([nvcc(), *ARCH, "-O3", "-std=c++17", "--expt-relaxed-constexpr", "-shared", "-Xcompiler", "-fPIC",
                        "-I", str(csrc), str(SRC), "-o", str(LIB)], check=True)
    return C.CDLL(str(LIB))


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_modulus_and_ratio_round_as_square_root_and_division(dtype):
    rng = np.random.default_rng(1)
    n = 1 << 20
    span = 29 if dtype == np.float32 else 270
    power = (10.0 ** rng.uniform(-span, span, n)).astype(dtype)
    power[: n // 2] = 10.0 ** rng.uniform(-4, 8, n // 2)  # what far fields hold
    measured = (10.0 ** rng.uniform(-6, 6, n)).astype(dtype)
    measured[::7] = 0
    modulus, ratio = np.empty_like(power), np.empty_like(power)
    f = _lib().ratio_f32 if dtype == np.float32 else _lib().ratio_f64
    assert f(_p(power), _p(measured), n, _p(modulus), _p(ratio)) == 0
    root = np.sqrt(power)
    quotient = measured / root
    # one correction of an estimate within two units: at most one unit in the last place off, almost always none
    for got, want in ((modulus, root), (ratio, quotient)):
        off = np.abs(got - want) / np.spacing(np.abs(want))
        assert off.max() <= 1, off.max()
        assert np.mean(off > 0) <= 0.01, np.mean(off > 0)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_projection_of_every_kind_of_value(dtype):
    rng = np.random.default_rng(2)
    ordinary = rng.normal(size=(400, 4)) + 1j * rng.normal(size=(400, 4))
    z = ordinary.astype(np.complex64 if dtype == np.float32 else np.complex128)
    special = np.array([0, 1e-22, 1e-19j, 3e17, 1e19j, 1e-17 + 1e-17j] if dtype == np.float32 else
                       [0, 1e-160, 1e-150j, 3e138, 1e145j, 1e-142 + 1e-142j])
    for i in range(200):  # one special value in each of half the groups
        z[i, i % 4] = special[i % len(special)]
    measured = np.abs(rng.normal(size=z.shape)).astype(np.float32)
    measured[::5] = 0
    inv_n = dtype(1 / 16384)
    out, err = np.empty_like(z), np.empty(len(z))
    f = _lib().project_f32 if dtype == np.float32 else _lib().project_f64
    scale = C.c_float(inv_n) if dtype == np.float32 else C.c_double(inv_n)
    assert f(_p(z), _p(measured), len(z), scale, _p(out), _p(err)) == 0
    w = z.astype(np.clongdouble)
    mag = np.abs(w)
    # the general path forms |f|^2 in the working type, as every pass does: a subnormal or overflowing square is part of
    # the definition there
    with np.errstate(over="ignore", under="ignore"):
        square = z.real * z.real + z.imag * z.imag
    low, high = (1e-30, 1e30) if dtype == np.float32 else (1e-280, 1e280)
    mag = np.where((square > low) & (square < high), mag, np.sqrt(square).astype(np.longdouble))
    with np.errstate(divide="ignore", invalid="ignore"):
        expected = np.where(mag > 0, (measured / np.where(mag > 0, mag, 1) - 1) * w, measured) * np.longdouble(inv_n)
    eps = np.finfo(dtype).eps
    # |f|, its square, the quotient and two products: a few roundings of the larger of A / n and |f| / n
    assert np.all(np.abs(out - expected) <= 8 * eps * np.maximum(measured, mag) * np.longdouble(inv_n))
    terms = ((measured - mag) ** 2).sum(1)
    assert np.all(np.abs(err - terms) <= 16 * eps * (np.maximum(measured, mag) ** 2).sum(1))


def test_values_not_finite_take_the_general_path():
    z = np.array([[np.nan, 1, 2, 3], [np.inf, 1, 2, 3]], np.complex64)
    measured = np.ones(z.shape, np.float32)
    out, err = np.empty_like(z), np.empty(2)
    assert _lib().project_f32(_p(z), _p(measured), 2, C.c_float(1.0), _p(out), _p(err)) == 0
    assert out[0, 0] == 1 and np.allclose(out[:, 1:], [[0, -1, -2]] * 2)  # a modulus that is not positive becomes A
    assert np.isnan(err[0]) and np.isinf(err[1])
