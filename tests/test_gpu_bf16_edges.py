"""The split-BF16 pass where its schedule changes: one position, one more or fewer than one per SM, CTAs of different lengths;
and far fields that are exactly zero, alone and beside ordinary ones.  Against the FP64 oracle, to the form's 1e-4."""
import numpy as np
import pytest

from oracle import c_oracle
from tests import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count,blank", [(1, 0), (2, 0), (147, 0), (148, 0), (149, 0), (300, 0), (5, 400), (150, 150)])
def test_against_the_oracle(count, blank):
    import cubokit_b200 as cb
    s = scenes.raster_scene(scan=18, det=128, step=4, seed=21)
    amps = s["amplitudes"][:count].astype(np.float32)
    positions = s["positions"][:count]
    start = s["object"].copy()
    start[:blank] = 0  # windows in these rows have a zero exit wave
    o, p, e = c_oracle.reconstruct(amps, positions, start, s["probe"], iterations=2)
    r = cb.SingleslicePtychography.reconstruct(amps, positions, start, s["probe"], iterations=2, precision="split_bf16")
    assert np.linalg.norm(r.object - o) <= 1e-4 * np.linalg.norm(o)
    assert np.linalg.norm(r.probe - p) <= 1e-4 * np.linalg.norm(p)
    assert np.all(np.abs(r.errors - e) <= 1e-4 * e)
