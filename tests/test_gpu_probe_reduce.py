"""The sum of the position groups' probe gradients and the weights' maximum, at detectors of one to ten groups (a thread a pixel,
and eighths of the groups), against the FP64 C oracle."""
import numpy as np
import pytest

from oracle import c_oracle
from tests import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("rows,columns", [(140, 140), (150, 160), (168, 170), (180, 180), (192, 192), (256, 255), (500, 481)])
def test_probe_against_the_oracle(precision, rows, columns):
    import cubokit_b200 as cb
    s = scenes.raster_scene(scan=4, step=4, seed=6, shape=(rows, columns))
    # a start probe half the true one's size: the update is as large as the probe
    args = (s["amplitudes"].astype(np.float32), s["positions"], s["object"], 0.5 * s["probe"])
    o, p, e = c_oracle.reconstruct(*args, iterations=2)
    r = cb.SingleslicePtychography.reconstruct(*args, iterations=2, precision=precision)
    # the reference's Float-vs-Double bounds; round-off of the transforms with far-field pixels 1e-6 of the largest
    assert np.max(np.abs(r.object - o)) <= (1e-4 if precision == "fp32" else 1e-9)
    assert np.max(np.abs(r.probe - p)) <= (1e-5 if precision == "fp32" else 1e-9) * max(1.0, np.max(np.abs(p)))
    assert np.max(np.abs(p - args[3])) >= 0.05 * np.max(np.abs(p))
