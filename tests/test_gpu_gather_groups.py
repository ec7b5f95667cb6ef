"""The object gather with each tile's candidates split into groups (small objects, 128 positions and more): against the
FP64 oracle, and the same bits whatever the tile shape, in a batch and run to run."""
import numpy as np
import pytest

from oracle import numpy_oracle
from tests import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scan", [12, 16, 24])  # 2, 4 and 8 groups: positions / 64, at most 8
@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_groups(scan, precision):
    import cubokit_b200 as cb
    s = scenes.raster_scene(scan=scan, det=24, step=3, seed=4)
    args = (s["amplitudes"], s["positions"], s["object"], s["probe"])
    o, p, e = numpy_oracle.reconstruct(*args, iterations=2)
    runs = [cb.SingleslicePtychography.reconstruct(*args, iterations=2, precision=precision, gather_tile=tile)
            for tile in (0, 1, 2, 3, 0)]
    r = runs[0]
    # the reference's Float-vs-Double bounds; FP64 agrees with the oracle to round-off
    assert np.max(np.abs(r.object - o)) <= (1e-4 if precision == "fp32" else 1e-9)
    assert np.all(np.abs(r.errors - e) <= (1e-5 if precision == "fp32" else 1e-9) * e)
    for other in runs[1:]:
        assert np.array_equal(r.object, other.object) and np.array_equal(r.probe, other.probe)
    batch = cb.Batch([dict(amplitudes=s["amplitudes"], positions=s["positions"], object=s["object"], probe=s["probe"],
                           precision=precision)] * 2)
    batch.run(2)
    for i in range(2):
        bo, bp = batch.get_state(i)
        assert np.array_equal(bo, r.object) and np.array_equal(bp, r.probe)
    batch.close()
