"""The cubic shift in registers at the sizes where its layout changes: one segment a line, the most segments, several CTAs an SM,
warps with idle lanes, the last size that fits, the first that does not, and a cube 4 bytes off alignment.  Against the FP64
restatement, to the reference's 2e-6."""
import numpy as np
import pytest

from oracle import numpy_oracle as no

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,columns,count", [(16, 16, 700), (16, 512, 3), (512, 16, 3), (48, 80, 301), (96, 96, 150),
                                                (128, 128, 149), (112, 144, 5), (144, 128, 4), (144, 144, 2), (176, 80, 3)])
def test_against_the_oracle(rows, columns, count):
    import cubokit_b200 as cb
    import torch
    rng = np.random.default_rng(rows + columns)
    cube = (rng.standard_normal((count, rows, columns)) + 0.3).astype(np.float32)
    o_rows, o_cols = rng.uniform(-2.5 * rows, 2.5 * rows, count), rng.uniform(-2.5 * columns, 2.5 * columns, count)
    o_rows[0], o_cols[0] = 0.0, columns - 1.0
    ref = no.prepare_amplitudes(cube, o_rows, o_cols, "cubicSpline")
    flat = torch.empty(cube.size + 1, device="cuda")
    flat[1:] = torch.from_numpy(cube).reshape(-1)
    shifted = flat[1:].view(cube.shape)
    for source in (torch.from_numpy(cube).cuda(), shifted):
        a = cb.PtychographyPreparation.amplitudes(source, (o_rows, o_cols), shift="cubicSpline")
        got = (a.values.cpu().numpy() if hasattr(a.values, "cpu") else a.values).reshape(cube.shape)
        assert np.max(np.abs(got - ref.values)) <= 2e-6 * max(1.0, np.max(ref.values))
        assert abs(a.mean_intensity - ref.mean_intensity) <= 1e-10 * max(1.0, abs(ref.mean_intensity))
        assert abs(a.clipped_mean_intensity - ref.clipped_mean_intensity) <= 1e-10 * ref.clipped_mean_intensity


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_not_finite_is_refused(value):
    import cubokit_b200 as cb
    cube = np.ones((3, 64, 96), np.float32)
    cube[1, 63, 95] = value
    with pytest.raises(cb.PtychographyError):
        cb.PtychographyPreparation.amplitudes(cube, (0.25, 0.5), shift="cubicSpline")
