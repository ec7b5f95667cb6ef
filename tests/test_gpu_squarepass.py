"""The compile-time 64 x 64 and 96 x 96 FP32 position pass against the FP64 C oracle: windows inside the object, touching
its edges and wrapping around them, whole-pixel and fractional positions."""
import numpy as np
import pytest

from oracle import c_oracle
from tests import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("det", [64, 96])
@pytest.mark.parametrize("wrapped", [False, True])
def test_against_the_oracle(det, wrapped):
    import cubokit_b200 as cb
    # the raster's windows run from edge to edge of the object; the other scene's reach over its first row and column
    s = scenes.nonsquare_scene(det, det, det + 60) if wrapped else scenes.raster_scene(scan=4, det=det, step=4, seed=3)
    amps = s["amplitudes"].astype(np.float32)
    o, p, e = c_oracle.reconstruct(amps, s["positions"], s["object"], s["probe"], iterations=3)
    r = cb.SingleslicePtychography.reconstruct(amps, s["positions"], s["object"], s["probe"], iterations=3)
    # the reference's Float-vs-Double bounds
    assert np.max(np.abs(r.object - o)) <= 1e-4
    assert np.max(np.abs(r.probe - p)) <= 1e-5 * max(1.0, np.max(np.abs(p)))
    assert np.all(np.abs(r.errors - e) <= 1e-5 * e)
