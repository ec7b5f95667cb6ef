"""The FP32 pass through global memory at the sizes where its line plans change: one, two and three stages, ragged last
blocks of lines, the prime radices above 13, and sides that take the direct DFT beside a planned one."""
import numpy as np
import pytest

from oracle import c_oracle
from tests import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,columns", [(128, 225), (225, 128), (288, 64), (64, 288), (128, 248), (248, 72), (96, 211),
                                          (211, 96), (1200, 16), (16, 1200), (320, 96)])
def test_against_the_oracle(rows, columns):
    import cubokit_b200 as cb
    s = scenes.raster_scene(scan=3, step=4, seed=6, shape=(rows, columns))
    amps = s["amplitudes"].astype(np.float32)
    positions = s["positions"] + np.array([[0.25, -0.3]]) * (np.arange(9)[:, None] % 2)
    o, p, e = c_oracle.reconstruct(amps, positions, s["object"], s["probe"], iterations=2)
    r = cb.SingleslicePtychography.reconstruct(amps, positions, s["object"], s["probe"], iterations=2)
    # the reference's Float-vs-Double bounds
    assert np.max(np.abs(r.object - o)) <= 1e-4
    assert np.max(np.abs(r.probe - p)) <= 1e-5 * max(1.0, np.max(np.abs(p)))
    assert np.all(np.abs(r.errors - e) <= 1e-5 * e)
