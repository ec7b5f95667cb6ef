"""The any-size shared-memory position pass (in-place digit-reversed line transforms) against the FP64 C oracle, at the
sizes where its plans change: one, two and three stages a side, every radix class, odd pitches, the wide primes, planes
near one CTA's limit, and the lengths it leaves to the run-time Stockham plan."""
import numpy as np
import pytest

from oracle import c_oracle, numpy_oracle
from tests import scenes

pytestmark = pytest.mark.gpu

# rows x columns: one stage (16, 13, 2), two (120 = 10 12, 112 = 8 14, 81 = 9 9), three (168 = 4 6 7), primes above 13
# (29, 31 and 124 = 4 31), the largest FP32 plane (128 x 128), and a prime above 31 (37: the run-time plan)
SIZES = [(16, 13), (2, 15), (6, 10), (120, 112), (112, 120), (81, 49), (168, 20), (22, 165), (31, 29), (124, 60),
         (128, 126), (37, 24), (64, 96)]


def _scene(rows, columns):
    return scenes.nonsquare_scene(rows, columns, max(rows, columns) + 60)


@pytest.mark.parametrize("rows,columns", SIZES)
def test_fp32_against_the_oracle(rows, columns):
    import cubokit_b200 as cb
    s = _scene(rows, columns)
    amps = s["amplitudes"].astype(np.float32)
    o, p, e = c_oracle.reconstruct(amps, s["positions"], s["object"], s["probe"], iterations=3)
    r = cb.SingleslicePtychography.reconstruct(amps, s["positions"], s["object"], s["probe"], iterations=3)
    # the reference's Float-vs-Double bounds
    assert np.max(np.abs(r.object - o)) <= 1e-4
    assert np.max(np.abs(r.probe - p)) <= 1e-5 * max(1.0, np.max(np.abs(p)))


@pytest.mark.parametrize("rows,columns", [s for s in SIZES if s[0] * s[1] <= 12288])
def test_fp64_against_the_oracles(rows, columns):
    """Held to how far the two FP64 restatements (C and NumPy, whose transforms differ) are from each other on the same
    input: far fields near zero make some of these scenes amplify round-off by up to 1e7."""
    import cubokit_b200 as cb
    s = _scene(rows, columns)
    amps = s["amplitudes"].astype(np.float32)
    args = (amps, s["positions"], s["object"], s["probe"])
    o, p, e = c_oracle.reconstruct(*args, iterations=3)
    on, pn, en = numpy_oracle.reconstruct(*args, iterations=3)
    runs = [cb.SingleslicePtychography.reconstruct(*args, iterations=3, precision="fp64") for _ in range(2)]
    r = runs[0]
    assert np.max(np.abs(r.object - o)) <= 1e-12 + 4 * np.max(np.abs(on - o))
    assert np.max(np.abs(r.probe - p)) <= 1e-12 + 4 * np.max(np.abs(pn - p))
    assert np.allclose(r.errors, e, rtol=1e-9, atol=0)
    assert np.array_equal(r.object, runs[1].object) and np.array_equal(r.errors, runs[1].errors)


@pytest.mark.parametrize("rows,columns", SIZES)
def test_fp32_errors_and_bits(rows, columns):
    """The squared residual, summed over CTAs of 128 to 1024 threads: with far fields off by d of the amplitudes' size it is
    off by at most 2 d sqrt(e) for a residual of e (both over the amplitudes' energy), d = 5e-7 for FP32 transforms of up to
    16,384 samples.  Twice the same bits."""
    import cubokit_b200 as cb
    s = scenes.raster_scene(scan=4, step=3, seed=5, shape=(rows, columns))
    args = (s["amplitudes"].astype(np.float32), s["positions"], s["object"], s["probe"])
    e = c_oracle.reconstruct(*args, iterations=3)[2]
    first, second = (cb.SingleslicePtychography.reconstruct(*args, iterations=3) for _ in range(2))
    assert np.all(np.abs(first.errors - e) <= 1e-6 * np.sqrt(e))
    assert np.array_equal(first.errors, second.errors) and np.array_equal(first.object, second.object)
    assert np.array_equal(first.probe, second.probe)
