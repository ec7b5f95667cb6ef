"""The generic variant's position pass (Stockham stages, square root and division) is another kernel than the default one at
every size that has a faster one: the results agree to round-off and are not the same bits.  In a batch it runs as alone."""
import numpy as np
import pytest

from tests import golden_cases as gc
from tests import scenes

pytestmark = pytest.mark.gpu


def _run(s, **more):
    import cubokit_b200 as cb
    return cb.SingleslicePtychography.reconstruct(s["amplitudes"], s["positions"], s["object"], s["probe"], iterations=2,
                                                  step_size=0.5, **more)


@pytest.mark.parametrize("precision,rows,columns", [
    ("fp32", 64, 64), ("fp32", 96, 96), ("fp32", 120, 112), ("fp32", 16, 13), ("fp32", 62, 29), ("fp32", 128, 128),
    ("fp64", 100, 90), ("fp64", 16, 13), ("fp64", 128, 96)])
def test_generic_agrees_and_is_another_kernel(precision, rows, columns):
    s = scenes.raster_scene(scan=3, step=5, seed=3, shape=(rows, columns))
    a, b = (_run(s, precision=precision, variant=v) for v in ("auto", "generic"))
    # FP64: round-off, turned into up to 1e-9 of its own phase by a far-field pixel 1e-6 of the largest
    tolerance = 2e-5 if precision == "fp32" else 1e-9
    assert np.max(np.abs(a.object - b.object)) <= tolerance
    assert gc.complex_gap(a.probe, b.probe) <= tolerance
    assert np.all(np.abs(a.errors - b.errors) <= (1e-5 if precision == "fp32" else 1e-9) * b.errors)
    assert not np.array_equal(a.object, b.object)


def test_generic_items_of_a_batch():
    """64 x 64 items of both variants: the default ones share a grouped launch, the generic one has its own."""
    import cubokit_b200 as cb
    s = scenes.raster_scene(scan=4, det=64, step=4, seed=7)
    variants = ["auto", "generic", "auto"]
    batch = cb.Batch([dict(amplitudes=s["amplitudes"], positions=s["positions"], object=s["object"], probe=s["probe"],
                           step_size=0.5, precision="fp32", variant=v) for v in variants])
    batch.run(2)
    for i, v in enumerate(variants):
        r = _run(s, precision="fp32", variant=v)
        o, p = batch.get_state(i)
        assert np.array_equal(o, r.object) and np.array_equal(p, r.probe), (i, v)
