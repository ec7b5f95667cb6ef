"""The shifted-probe table in one launch (folded in-place inverse transforms) against NumPy, through the forward loss of
fractional positions: the sizes where its plan changes (fold 1, 2, 3, 8 and a fold by a prime factor of the rows; one,
two and three stages a line; odd sides) and those it leaves to the line transforms."""
import numpy as np
import pytest

from oracle import numpy_oracle
from tests import scenes

pytestmark = pytest.mark.gpu

SIZES = [(40, 48), (128, 128), (2, 15), (16, 13), (160, 96), (256, 256), (63, 45), (192, 200), (34, 40), (40, 34)]


def _loss(s, positions):
    rows, columns = s["probe"].shape
    o = s["object"]
    rr, cc = (numpy_oracle.round_half_even(positions[:, i]) for i in (0, 1))
    idx = numpy_oracle.patch_indices(rows, columns, *o.shape, rr.astype(np.int64), cc.astype(np.int64))
    shifted = numpy_oracle.shifted_probes(np.fft.fft2(s["probe"]), positions[:, 0] - rr, positions[:, 1] - cc)
    far = np.fft.fft2(shifted * o.reshape(-1)[idx].reshape(shifted.shape))
    return float(np.sum((np.abs(far) - s["amplitudes"].reshape(far.shape)) ** 2))


@pytest.mark.parametrize("rows,columns", SIZES)
def test_loss_of_fractional_positions(rows, columns):
    import cubokit_b200 as cb
    s = scenes.raster_scene(scan=3, step=4, seed=5, shape=(rows, columns))
    rng = np.random.default_rng(8)
    positions = s["positions"] + rng.uniform(-0.5, 0.5, s["positions"].shape)
    positions[4] = s["positions"][4]  # one whole-pixel position: class 0
    expected = _loss(s, positions)
    # FP64: round-off of a few thousand terms; FP32: transforms in single precision
    for precision, rtol in (("fp64", 1e-11), ("fp32", 2e-5)):
        plan = cb.Plan(s["amplitudes"].astype(np.float32), positions, s["object"].shape, s["probe"].shape,
                       precision=precision)
        plan.set_state(s["object"], s["probe"])
        assert abs(plan.forward() - expected) <= rtol * expected, precision
        plan.close()
