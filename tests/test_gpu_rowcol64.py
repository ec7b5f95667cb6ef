"""FP64 planes by row and column launches (``rowcol64.cu``) against the batched line transforms of the generic variant, engine by
engine, where the plans change: two and three stages, odd and prime last radices, 128 on either side, ragged last CTAs, the most
states, and a side left to the line transforms.

The same arithmetic in another order.  A pixel whose far field is 1e-6 of the largest turns the transforms' round-off, about 1e-15 of
the largest, into 1e-9 of its own phase; results are held to that."""
import numpy as np
import pytest

from tests import golden_cases as gc
from tests import scenes

pytestmark = pytest.mark.gpu

TOL = 1e-9
SIZES = [(24, 36), (45, 63), (128, 45), (18, 128), (26, 169), (288, 40), (40, 288), (130, 17)]


def _scene(rows, columns):
    s = scenes.raster_scene(scan=3, step=5, seed=3, shape=(rows, columns))
    s["start"] = s["positions"] + np.array([[0.25, -0.4]]) * (np.arange(9)[:, None] % 2)
    return s


def _compare(s, make, object_, probe):
    import cubokit_b200 as cb
    out = []
    for variant in ("auto", "auto", "generic"):
        plan = cb.Plan(s["amplitudes"], s["start"], s["object"].shape, s["probe"].shape, variant=variant, step_size=0.5, **make(cb))
        plan.set_state(object_, probe)
        e = plan.iterate(2)
        out.append((*plan.get_state(), e))
        plan.close()
    first, second, generic = out
    assert all(np.array_equal(a, b) for a, b in zip(first, second))
    assert gc.complex_gap(first[0], generic[0]) < TOL
    assert gc.complex_gap(first[1], generic[1]) < TOL
    assert gc.gap(first[2], generic[2]) < TOL


@pytest.mark.parametrize("rows,columns,states", [(*size, 3) for size in SIZES] + [(128, 128, 11), (128, 128, 12), (24, 36, 16)])
def test_mixed_states(rows, columns, states):
    import cubokit_b200 as cb
    s = _scene(rows, columns)
    probes = cb.MixedstatePtychography.initial_probes(s["probe"] / np.sqrt(states), states, seed=4)
    _compare(s, lambda cb: dict(mixed_states=states), s["object"], probes)


@pytest.mark.parametrize("rows,columns", SIZES)
def test_multislice(rows, columns):
    s = _scene(rows, columns)
    obj = np.stack([s["object"] * np.exp(0.03j * i) for i in range(3)])
    ms = dict(slices=3, slice_thicknesses=[30.0, 50.0], wavelength=0.0197, row_sampling=0.45, column_sampling=0.5)
    _compare(s, lambda cb: dict(multislice=ms), obj, s["probe"])


@pytest.mark.parametrize("rows,columns", SIZES)
def test_position_correction(rows, columns):
    s = _scene(rows, columns)
    _compare(s, lambda cb: dict(precision="fp64", position_correction=cb.PtychographyPositionCorrection(
        step_size=0.5, max_update_distance=0.3, row_sampling=0.5, column_sampling=0.5)), s["object"], s["probe"])


@pytest.mark.parametrize("rows,columns", [(128, 128), (130, 112), (160, 96), (288, 45)])
def test_single_slice(rows, columns):
    s = _scene(rows, columns)
    _compare(s, lambda cb: dict(precision="fp64"), s["object"], s["probe"])


@pytest.mark.parametrize("slices", [1, 2, 4, 5])
@pytest.mark.parametrize("rows,columns", [(24, 36), (128, 40), (40, 288)])
def test_multislice_depths(rows, columns, slices):
    """No gap, one, and several (a wave's place is taken over by a spectrum once its gather has read it)."""
    s = _scene(rows, columns)
    obj = np.stack([s["object"] * np.exp(0.02j * i) for i in range(slices)])
    ms = dict(slices=slices, slice_thicknesses=[20.0 + 5 * i for i in range(slices - 1)], wavelength=0.0197,
              row_sampling=0.45, column_sampling=0.5)
    _compare(s, lambda cb: dict(multislice=ms), obj, s["probe"])
