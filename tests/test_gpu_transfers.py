"""Host arrays to and from the device: pageable, page-locked and device amplitudes, and the interleaved complex calls
beside the ones with a real and an imaginary plane."""
import ctypes as C

import numpy as np
import pytest

from tests import scenes

pytestmark = pytest.mark.gpu


def _scene():
    # 840 x 790 object pixels: two ranges of values, converted by two threads
    rng = np.random.default_rng(3)
    probe = scenes.raster_scene(scan=2, det=40, step=4, seed=5)["probe"]
    positions = np.stack([rng.integers(20, 820, 1437), rng.integers(20, 770, 1437)], 1).astype(np.float64)
    amplitudes = rng.uniform(0, 2, (1437, 40, 40)).astype(np.float32)
    obj = np.exp(1j * rng.normal(0, 0.1, (840, 790)))
    return amplitudes, positions, obj, probe


def test_pageable_amplitudes_equal_device_ones():
    import torch
    import cubokit_b200 as cb
    amplitudes, positions, obj, probe = _scene()
    losses = []
    for a in (amplitudes, torch.from_numpy(amplitudes).cuda(), torch.from_numpy(amplitudes).pin_memory().numpy()):
        plan = cb.Plan(a, positions, obj.shape, probe.shape)
        plan.set_state(obj, probe)
        losses.append(plan.forward())
        plan.close()
    assert losses[0] == losses[1] == losses[2]


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_interleaved_and_plane_calls_agree(precision):
    import cubokit_b200 as cb
    amplitudes, positions, obj, probe = _scene()
    plan = cb.Plan(amplitudes, positions, obj.shape, probe.shape, precision=precision)
    lib, h = plan.ctx.lib, plan.handle
    ptr = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))  # noqa: E731

    def planes(z):
        return np.ascontiguousarray(z.real), np.ascontiguousarray(z.imag)

    plan.set_state(obj, probe)
    held = obj.astype(np.complex64) if precision == "fp32" else obj
    o, p = plan.get_state()
    assert np.array_equal(o, held.astype(np.complex128)) and np.array_equal(p, probe)
    (ore, oim), (pre, pim) = planes(obj), planes(probe)
    assert lib.cubo_ptycho_plan_set_state(h, ptr(ore), ptr(oim), ptr(pre), ptr(pim)) == 0
    ore[:], oim[:], pre[:], pim[:] = 0, 0, 0, 0
    assert lib.cubo_ptycho_plan_get_state(h, ptr(ore), ptr(oim), ptr(pre), ptr(pim)) == 0
    assert np.array_equal(ore + 1j * oim, o) and np.array_equal(pre + 1j * pim, p)
    loss, go, gp = plan.backward()
    l2 = C.c_double(0)
    assert lib.cubo_ptycho_plan_backward(h, 0, C.byref(l2), ptr(ore), ptr(oim), ptr(pre), ptr(pim)) == 0
    assert l2.value == loss and np.array_equal(ore + 1j * oim, go) and np.array_equal(pre + 1j * pim, gp)
    # a value that is not finite anywhere is refused and leaves the state
    for bad in (np.nan, np.inf * 1j):
        broken = obj.copy()
        broken[-1, -1] = bad
        with pytest.raises(cb.PtychographyError):
            plan.set_state(broken, probe)
    again, _ = plan.get_state()
    assert np.array_equal(again, o)
    plan.close()
