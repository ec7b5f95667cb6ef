"""The work a user of this package gives it, as cases that can be timed: whole reconstructions from host arrays,
iterations on a device-resident plan in every form (FP32, split-BF16, FP64) and at every class of detector size, the
adjoint pair, position correction, the mixed-state and multislice engines, batches and the amplitude preprocessing.

A case is a dict of plain values.  ``prepare(case, seed)`` makes what a program holds before the call (inputs from the
seed alone, and the plan or batch it keeps), ``run(state)`` is one pass through the public entry points, ``work(case)``
the bytes and flops the pass cannot do without, ``exact(case, seed)`` the same results in 64 bits by plain torch.

Every dataset is the synthetic recipe of ``cubokit_b200/synthetic.py`` (unit-amplitude phase object, 300 kV probe,
square-root Poisson counts, 4 px raster), drawn here with torch so that the inputs do not depend on the package.
"""
import math

import numpy as np
import torch

import cubokit_b200 as cb

WAVELENGTH = 0.019687  # Å, 300 kV


def listed():
    return [
        # A quick look at the microscope: a small scan on a binned detector, host arrays in and out, the default eight
        # iterations.  Upload, plan creation, launches and read-back are most of it.
        dict(name="reconstruct_fp32_64_scan24", kind="reconstruct", precision="fp32", rows=64, columns=64,
             scan_rows=24, scan_columns=24, step=4, rotation=0.0, iterations=8, dose=1e4),
        # The benchmark's mid detector in FP32, a raster along the object's axes.
        dict(name="adjoint_fp32_96_scan48", kind="adjoint", precision="fp32", rows=96, columns=96, scan_rows=48,
             scan_columns=48, step=4, rotation=0.0, iterations=1, dose=1e5),
        # What an instrument delivers: the scan is rotated against the detector, so no position is a whole pixel and
        # every one has its own shifted probe.
        dict(name="iterate_fp32_128_rotated", kind="iterate", precision="fp32", rows=128, columns=128, scan_rows=56,
             scan_columns=60, step=4, rotation=7.5, iterations=8, dose=1e5),
        # The FP32 benchmark workload: 128^2 scan, 128^2 detector.
        dict(name="iterate_fp32_128_scan128", kind="iterate", precision="fp32", rows=128, columns=128, scan_rows=128,
             scan_columns=128, step=4, rotation=0.0, iterations=8, dose=1e5),
        # The headline workload: 256^2 scan, 128^2 detector on the tensor cores.
        dict(name="iterate_bf16_128_scan256", kind="iterate", precision="split_bf16", rows=128, columns=128,
             scan_rows=256, scan_columns=256, step=4, rotation=0.0, iterations=8, dose=1e5),
        # An unbinned detector: planes too large for one thread block's shared memory.
        dict(name="iterate_fp32_256_scan64", kind="iterate", precision="fp32", rows=256, columns=256, scan_rows=64,
             scan_columns=64, step=4, rotation=0.0, iterations=4, dose=1e5),
        # A detector cropped around the bright field: neither square nor a power of two.
        dict(name="iterate_fp32_120x112", kind="iterate", precision="fp32", rows=120, columns=112, scan_rows=60,
             scan_columns=53, step=4, rotation=0.0, iterations=8, dose=1e5),
        # Refinement of the scan: position correction, which runs in FP64, from amplitudes already on the device.
        dict(name="positions_fp64_128_scan48", kind="positions", precision="fp64", rows=128, columns=128,
             scan_rows=48, scan_columns=48, step=4, rotation=0.0, iterations=4, dose=1e5),
        # Partial coherence: four probe states.
        dict(name="mixed_fp64_128_scan40", kind="mixed", precision="fp64", rows=128, columns=128, scan_rows=40,
             scan_columns=40, step=4, rotation=0.0, iterations=4, dose=1e5, states=4),
        # A thick specimen: four slices 20 Å apart.
        dict(name="multislice_fp64_128_scan40", kind="multislice", precision="fp64", rows=128, columns=128,
             scan_rows=40, scan_columns=40, step=4, rotation=0.0, iterations=4, dose=1e5, slices=4),
        # A tilt or time series: independent reconstructions of mixed sizes advanced together.
        dict(name="batch_fp32_12", kind="batch", precision="fp32", items=12, scan_low=24, scan_high=72, step=4,
             iterations=8, dose=1e5),
        # Every reconstruction's first step: raw patterns to corner-centred amplitudes, periodic cubic spline.
        dict(name="prepare_cubic_128", kind="prepare", shift="cubicSpline", rows=128, columns=128, count=16384,
             per_position=False, dose=1e5),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    """One more case of the same ranges: scans of 12 to 96 positions a side, detectors of 24 to 288 pixels a side."""
    kind = rng.choice(["reconstruct", "adjoint", "iterate", "iterate", "iterate", "iterate", "positions", "mixed",
                       "multislice", "batch", "prepare", "prepare"])
    if kind == "batch":
        low = _log_int(rng, 12, 32)
        return dict(kind=kind, precision="fp32", items=rng.randint(3, 16), scan_low=low,
                    scan_high=min(72, low + rng.randint(4, 40)), step=rng.randint(3, 6), iterations=rng.randint(2, 8),
                    dose=1e5)
    if kind == "prepare":
        shift = rng.choice(["cubicSpline", "bilinear"])
        rows = rng.choice([64, 96, 128, rng.randint(24, 156)])
        columns = rows if rng.random() < 0.5 else rng.randint(24, 156)
        return dict(kind=kind, shift=shift, rows=rows, columns=columns, count=_log_int(rng, 256, 12000),
                    per_position=rng.random() < 0.5, dose=1e5)
    precision = "fp32"
    if kind == "iterate":
        precision = rng.choice(["fp32", "fp32", "fp32", "split_bf16", "fp64"])
    elif kind in ("positions", "mixed", "multislice"):
        precision = "fp64"
    if precision == "split_bf16":
        rows = columns = 128
    else:
        ceiling = 288 if precision == "fp32" else 128
        rows = rng.choice([64, 96, 128, _log_int(rng, 24, ceiling), _log_int(rng, 24, ceiling)])
        columns = rows if rng.random() < 0.5 else _log_int(rng, 24, ceiling)
    scan_rows, scan_columns = _log_int(rng, 12, 96), _log_int(rng, 12, 96)
    heavy = dict(positions=4, mixed=12, multislice=12).get(kind, 8 if precision == "fp64" else 1)
    while scan_rows * scan_columns * rows * columns * heavy > 1.5e8:
        scan_rows, scan_columns = max(8, scan_rows * 3 // 4), max(8, scan_columns * 3 // 4)
    case = dict(kind=kind, precision=precision, rows=rows, columns=columns, scan_rows=scan_rows,
                scan_columns=scan_columns, step=rng.randint(2, 6),
                rotation=rng.choice([0.0, 0.0, round(rng.uniform(-20, 20), 3)]),
                iterations=1 if kind == "adjoint" else rng.randint(2, 8), dose=1e5)
    if kind == "adjoint":
        case["rotation"] = 0.0
    if kind == "mixed":
        case["states"] = rng.randint(2, 4)
    if kind == "multislice":
        case["slices"] = rng.randint(2, 4)
    return case


# ------------------------------------------------------------------------------------------------ inputs

def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) % (1 << 62))
    return g


def _frequency(n):
    return torch.fft.fftfreq(n, dtype=torch.float64, device="cuda")


def _corner(n):
    k = torch.arange(n, device="cuda")
    return torch.where(k < (n + 1) // 2, k, k - n)


def _probe(rows, columns, dose):
    """The 20 mrad, 100 Å defocus probe at 64 / N mrad per pixel, its pattern holding `dose` counts."""
    kr, kc = (64e-3 * _frequency(n) / WAVELENGTH for n in (rows, columns))
    k = torch.sqrt(kr[:, None] ** 2 + kc[None, :] ** 2)
    alpha = k * WAVELENGTH * 1e3
    soft = torch.clamp((21.0 - alpha) / 2.0, 0.0, 1.0)
    chi = math.pi * WAVELENGTH * 100.0 * k ** 2
    p = torch.fft.ifft2(soft * torch.exp(-1j * chi))
    return p * math.sqrt(dose / float((rows * columns * (p.abs() ** 2).sum())))


def _phases(rows, columns, g):
    noise = torch.randn(rows, columns, dtype=torch.float64, device="cuda", generator=g)
    k2 = _frequency(rows)[:, None] ** 2 + _frequency(columns)[None, :] ** 2
    f = torch.fft.ifft2(torch.fft.fft2(noise) * torch.exp(-2 * (math.pi * 3.0) ** 2 * k2)).real
    return (f - f.min()) / (f.max() - f.min()) * 0.5


def _positions(case):
    i = torch.arange(case["scan_rows"], dtype=torch.float64)[:, None] * case["step"]
    j = torch.arange(case["scan_columns"], dtype=torch.float64)[None, :] * case["step"]
    y, x = (i + 0 * j).reshape(-1), (0 * i + j).reshape(-1)
    if case["rotation"]:
        a = math.radians(case["rotation"])
        y0, x0 = y - y.mean(), x - x.mean()
        y, x = y.mean() + y0 * math.cos(a) - x0 * math.sin(a), x.mean() + y0 * math.sin(a) + x0 * math.cos(a)
    return torch.stack([y + case["rows"] // 2, x + case["columns"] // 2], 1).cuda()


def _windows(centres, rows, columns, object_rows, object_columns):
    """The flat object index of every detector pixel of every position, (P, rows, columns)."""
    rr = torch.remainder(centres[:, 0, None] + _corner(rows), object_rows)
    cc = torch.remainder(centres[:, 1, None] + _corner(columns), object_columns)
    return rr[:, :, None] * object_columns + cc[:, None, :]


def _chunks(total, n, planes=1):
    size = max(1, (1 << 25) // (n * planes))
    return [(b, min(total, b + size)) for b in range(0, total, size)]


def _shifted(spectrum, fractions):
    """``ifft2(spectrum * ramp)`` per position; (..., P, R, C) for spectra (..., R, C)."""
    fr, fc = _frequency(spectrum.shape[-2]), _frequency(spectrum.shape[-1])
    ramp = (torch.exp(-2j * math.pi * fr * fractions[:, 0, None])[:, :, None]
            * torch.exp(-2j * math.pi * fc * fractions[:, 1, None])[:, None, :])
    return torch.fft.ifft2(spectrum[..., None, :, :] * ramp)


def _inputs(case, seed):
    """Amplitudes (device, Float32), positions, start object(s), start probe(s), as device tensors."""
    g = _generator(seed, 1)
    rows, columns = case["rows"], case["columns"]
    object_rows = case["scan_rows"] * case["step"] + rows
    object_columns = case["scan_columns"] * case["step"] + columns
    truth = torch.exp(1j * _phases(object_rows, object_columns, g))
    probe = _probe(rows, columns, case["dose"])
    positions = _positions(case)
    measured = positions
    if case["kind"] == "positions":  # the data come from places up to 0.4 px off the recorded ones
        measured = positions + 0.8 * (torch.rand(positions.shape, dtype=torch.float64, device="cuda", generator=g) - 0.5)
    centres = torch.round(measured)
    windows = centres.long()
    fractions = measured - centres
    spectrum = torch.fft.fft2(probe)
    whole = bool((fractions == 0).all())
    amplitudes = torch.empty(len(positions), rows, columns, dtype=torch.float32, device="cuda")
    flat = truth.reshape(-1)
    for b, e in _chunks(len(positions), rows * columns):
        s = probe[None] if whole else _shifted(spectrum, fractions[b:e])
        wave = torch.fft.fft2(s * flat[_windows(windows[b:e], rows, columns, object_rows, object_columns)])
        intensity = (wave.real ** 2 + wave.imag ** 2).float()
        amplitudes[b:e] = torch.sqrt(torch.poisson(intensity, generator=g))
    slices = case.get("slices", 1)
    shape = (slices, object_rows, object_columns) if slices > 1 else (object_rows, object_columns)
    start = torch.exp(0.02j * torch.randn(shape, dtype=torch.float64, device="cuda", generator=g))
    probes = probe
    if case.get("states"):
        fr, fc = _frequency(rows)[:, None], _frequency(columns)[None, :]
        states = [probe]
        for _ in range(1, case["states"]):
            u = torch.rand(2, dtype=torch.float64, device="cuda", generator=g) - 0.5
            states.append(states[-1] * 0.5 * torch.exp(-2j * math.pi * (u[0] * fr + u[1] * fc)))
        probes = torch.stack(states)
    return dict(amplitudes=amplitudes, positions=positions, object=start, probe=probes)


def _items(case, seed):
    """The reconstructions of a batch: scan sides over the case's range, detectors in turn 64, 96 and 128."""
    count = case["items"]
    items = []
    for i in range(count):
        scan = case["scan_low"] + (case["scan_high"] - case["scan_low"]) * ((i * 5) % count) // max(1, count - 1)
        items.append(dict(kind="iterate", precision=case["precision"], rows=(64, 96, 128)[i % 3],
                          columns=(64, 96, 128)[i % 3], scan_rows=scan, scan_columns=max(8, scan - i % 4),
                          step=case["step"], rotation=0.0, iterations=case["iterations"], dose=case["dose"]))
    return [(c, int(seed) * 64 + i) for i, c in enumerate(items)]


def _patterns(case, seed):
    """Raw diffraction patterns: a soft disk of counts off the corner, its origin per position or one for all."""
    g = _generator(seed, 2)
    count, rows, columns = case["count"], case["rows"], case["columns"]
    jitter = torch.rand(count, 2, dtype=torch.float64, device="cuda", generator=g)
    origin = torch.tensor([rows / 2 + 0.3, columns / 2 - 0.45], dtype=torch.float64, device="cuda")
    origins = origin + 4 * (jitter - 0.5) if case["per_position"] else origin.expand(count, 2)
    cube = torch.empty(count, rows, columns, dtype=torch.float32, device="cuda")
    y = torch.arange(rows, device="cuda", dtype=torch.float32)
    x = torch.arange(columns, device="cuda", dtype=torch.float32)
    for b, e in _chunks(count, rows * columns):
        o = origins[b:e].float()
        r = torch.sqrt((y - o[:, 0, None])[:, :, None] ** 2 + (x - o[:, 1, None])[:, None, :] ** 2)
        disk = torch.sigmoid(min(rows, columns) * 0.31 - r) + 1e-3
        mean = disk * (case["dose"] / disk.sum(dim=(1, 2), keepdim=True))
        cube[b:e] = torch.poisson(mean, generator=g)
    return cube, origins


# ------------------------------------------------------------------------------------------------ prepare and run

def _host(x):
    return x.cpu().numpy()


def _multislice(case):
    return dict(slices=case["slices"], slice_thicknesses=[20.0] * (case["slices"] - 1), wavelength=WAVELENGTH,
                row_sampling=WAVELENGTH / 64e-3, column_sampling=WAVELENGTH / 64e-3)


def prepare(case, seed):
    kind = case["kind"]
    state = dict(case=case)
    if kind == "prepare":
        cube, origins = _patterns(case, seed)
        state["cube"] = cube
        state["out"] = torch.empty_like(cube)
        o = _host(origins)
        state["origins"] = (o[:, 0].copy(), o[:, 1].copy()) if case["per_position"] else (float(o[0, 0]), float(o[0, 1]))
        return state
    if kind == "batch":
        items = []
        for c, s in _items(case, seed):
            d = _inputs(c, s)
            items.append(dict(amplitudes=d["amplitudes"], positions=_host(d["positions"]), object=_host(d["object"]),
                              probe=_host(d["probe"]), precision=c["precision"]))
        state["starts"] = [(i["object"], i["probe"]) for i in items]
        state["batch"] = cb.Batch(items)
        return state
    d = _inputs(case, seed)
    state.update(object=_host(d["object"]), probe=_host(d["probe"]), positions=_host(d["positions"]))
    if kind == "reconstruct":
        state["amplitudes"] = _host(d["amplitudes"])
        return state
    state["amplitudes"] = d["amplitudes"]
    if kind == "positions":
        torch.cuda.synchronize()
        return state
    more = {}
    if kind == "mixed":
        more["mixed_states"] = case["states"]
    elif kind == "multislice":
        more["multislice"] = _multislice(case)
    else:
        more["precision"] = case["precision"]
    torch.cuda.synchronize()
    state["plan"] = cb.Plan(d["amplitudes"], state["positions"], state["object"].shape[-2:], state["probe"].shape[-2:],
                            **more)
    state["amplitudes"] = None
    return state


def _held(case, *arrays):
    """Results in the precision the form holds them in on the device (the interface hands every form out in doubles)."""
    if case["precision"] == "fp64":
        return tuple(arrays)
    return tuple(np.asarray(a).astype(np.complex64 if np.iscomplexobj(a) else np.float32) for a in arrays)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "prepare":
        r = cb.PtychographyPreparation.amplitudes(state["cube"], state["origins"], shift=case["shift"],
                                                  out=state["out"])
        return r.values, r.mean_intensity, r.clipped_mean_intensity
    if kind == "batch":
        batch = state["batch"]
        for i, (obj, probe) in enumerate(state["starts"]):
            batch.set_state(i, obj, probe)
        batch.run(case["iterations"])
        return [_held(case, *batch.get_state(i), batch.errors(i, case["iterations"])) for i in range(len(batch))]
    if kind == "reconstruct":
        r = cb.SingleslicePtychography.reconstruct(state["amplitudes"], state["positions"], state["object"],
                                                   state["probe"], iterations=case["iterations"],
                                                   precision=case["precision"])
        return _held(case, r.object, r.probe, r.errors)
    if kind == "positions":
        r = cb.SingleslicePtychography.reconstruct(state["amplitudes"], state["positions"], state["object"],
                                                   state["probe"], iterations=case["iterations"], precision="fp64",
                                                   position_correction=cb.PtychographyPositionCorrection(step_size=0.5))
        return r.object, r.probe, r.errors, r.positions
    plan = state["plan"]
    plan.set_state(state["object"], state["probe"])
    if kind == "adjoint":
        loss = plan.forward()
        again, grad_object, grad_probe = plan.backward()
        return _held(case, np.array([loss, again]), grad_object, grad_probe)
    errors = plan.iterate(case["iterations"])
    obj, probe = plan.get_state()
    return _held(case, obj, probe, errors)


# ------------------------------------------------------------------------------------------------ work

def _gd_work(case):
    n, count = case["rows"] * case["columns"], case["scan_rows"] * case["scan_columns"]
    objects = (case["scan_rows"] * case["step"] + case["rows"]) * (case["scan_columns"] * case["step"] + case["columns"])
    fractional = case["rotation"] != 0.0
    transforms = 2.0 * case.get("states", 1)
    if case.get("slices"):
        transforms = 2.0 + 4.0 * (case["slices"] - 1)
    if case["kind"] == "positions":
        transforms += 3.0
        fractional = True
    if fractional:
        transforms += 1.0
    value = 16 if case["precision"] == "fp64" else 8
    bytes_ = 4.0 * n * count + 2.0 * value * (objects * case.get("slices", 1) + n * case.get("states", 1))
    flops = count * (5.0 * transforms * n * math.log2(n) + 40.0 * n * case.get("states", 1) * case.get("slices", 1))
    return case["iterations"] * bytes_, case["iterations"] * flops


def work(case):
    if case["kind"] == "prepare":
        pixels = case["count"] * case["rows"] * case["columns"]
        return {"bytes": 8.0 * pixels, "flops": (60.0 if case["shift"] == "cubicSpline" else 12.0) * pixels}
    if case["kind"] == "batch":
        parts = [_gd_work(c) for c, _ in _items(case, 0)]
    else:
        parts = [_gd_work(case)]
    return {"bytes": sum(b for b, _ in parts), "flops": sum(f for _, f in parts)}


# ------------------------------------------------------------------------------------------------ 64-bit results

class _Sums:
    """Sums over the positions: the object's by scattering, FP64."""

    def __init__(self, objects, slices=1):
        self.grad = torch.zeros(slices, objects, 2, dtype=torch.float64, device="cuda")
        self.weight = torch.zeros(slices, objects, dtype=torch.float64, device="cuda")

    def add(self, slice_, index, waves, residuals):
        index = index.reshape(-1)
        self.grad[slice_].index_add_(0, index, torch.view_as_real(torch.conj(waves) * residuals).reshape(-1, 2))
        self.weight[slice_].index_add_(0, index, (waves.real ** 2 + waves.imag ** 2).expand_as(residuals).reshape(-1))


def _inverse(maximum):
    return 1 / torch.sqrt(1e-16 + maximum * maximum)  # normalisation minimum 1


def _capped(o):
    a = o.abs()
    return torch.where(a > 0, o * (torch.clamp(a, max=1.0) / torch.where(a > 0, a, 1.0)), torch.clamp(a, max=1.0) + 0j)


def _project(far, amplitudes):
    """The residual of one state's far field and the squared error."""
    mag = far.abs()
    error = ((amplitudes - mag) ** 2).sum()
    safe = torch.where(mag > 0, mag, 1.0)
    return torch.where(mag > 0, far * (amplitudes / safe - 1), amplitudes + 0j), error


def _orthogonal(p):
    """The eigenvectors of the states' Gram matrix by decreasing intensity (phases free)."""
    flat = p.reshape(p.shape[0], -1)
    values, vectors = torch.linalg.eigh(torch.conj(flat) @ flat.T)
    return (vectors.T @ flat)[torch.argsort(values, descending=True)].reshape(p.shape)


def _moved(before, after, spectrum, amplitudes, positions, shape):
    """One position-correction step of every position (2 x 2 least squares), no limits, step 0.5."""
    rows, columns = spectrum.shape
    out = positions.clone()
    for b, e in _chunks(len(positions), rows * columns, 4):
        centres = torch.round(positions[b:e])
        s = _shifted(spectrum, positions[b:e] - centres)

        def far(o, dy, dx):
            shift = torch.tensor([dy, dx], device="cuda")
            return torch.fft.fft2(s * o[_windows(centres.long() + shift, rows, columns, *shape)])

        f, fdx, fdy = far(before, 0, 0), far(after, 1, 0), far(after, 0, 1)
        difference = amplitudes[b:e].double() ** 2 - (f.real ** 2 + f.imag ** 2)
        dx = 2 * ((f.real - fdx.real) * f.real + (f.imag - fdx.imag) * f.imag)
        dy = 2 * ((f.real - fdy.real) * f.real + (f.imag - fdy.imag) * f.imag)
        total = lambda v: v.sum(dim=(1, 2))  # noqa: E731
        axx, axy, ayy, bx, by = (total(v) for v in (dx * dx, dx * dy, dy * dy, dx * difference, dy * difference))
        det = axx * ayy - axy * axy
        u = torch.stack([(ayy * bx - axy * by) / det, (axx * by - axy * bx) / det], 1) * 0.5
        out[b:e] -= torch.where(torch.isfinite(u).all(1, keepdim=True), u, 0.0)
    return out


def _reconstructed(case, seed, gradients_only=False):
    """Object, probe(s), errors and positions of the single-slice, mixed-state and position-correcting loops."""
    d = _inputs(case, seed)
    amplitudes, positions, o, p = d["amplitudes"], d["positions"], d["object"], d["probe"]
    shape, rows, columns = o.shape, case["rows"], case["columns"]
    o, n, count = o.reshape(-1), rows * columns, len(positions)
    mixed = case["kind"] == "mixed"
    p = p if mixed else p[None]
    energy = sum((amplitudes[b:e].double() ** 2).sum() for b, e in _chunks(count, n))
    errors = []
    for _ in range(case["iterations"]):
        centres = torch.round(positions)
        fractions = positions - centres
        whole = bool((fractions == 0).all())
        spectrum = torch.fft.fft2(p)
        sums = _Sums(o.numel())
        grad_p, weight_p, error = torch.zeros_like(p), torch.zeros(rows, columns, dtype=torch.float64, device="cuda"), 0.0
        for b, e in _chunks(count, n, len(p)):
            index = _windows(centres[b:e].long(), rows, columns, *shape)
            patch = o[index]
            s = p[:, None] if whole else _shifted(spectrum, fractions[b:e])
            far = torch.fft.fft2(s * patch)
            a = amplitudes[b:e].double()
            if mixed:
                mag = torch.sqrt((far.real ** 2 + far.imag ** 2).sum(0))
                error = error + ((a - mag) ** 2).sum()
                residual = torch.fft.ifft2(far * (a / mag - 1))
            else:
                residual, part = _project(far[0], a)
                error = error + part
                residual = torch.fft.ifft2(residual)[None]
            for st in range(len(p)):
                sums.add(0, index, s[st], residual[st])
            grad_p = grad_p + (torch.conj(patch) * residual).sum(1)
            weight_p = weight_p + (patch.real ** 2 + patch.imag ** 2).sum(0)
        if gradients_only:
            grad = torch.view_as_complex(sums.grad[0])
            return error, -2 * n * grad.reshape(shape), -2 * n * grad_p[0]
        before = o
        o = o + 0.5 * _inverse(sums.weight[0].max()) * torch.view_as_complex(sums.grad[0])
        if case["kind"] == "positions":
            positions = _moved(before, o, spectrum[0], amplitudes, positions, shape)
        o = _capped(o)
        p = p + 0.5 * _inverse(weight_p.max()) * grad_p
        if mixed:
            p = _orthogonal(p)
        errors.append(float(error / energy))
    return o.reshape(shape), (p if mixed else p[0]), np.array(errors), positions


def _sliced(case, seed):
    d = _inputs(case, seed)
    amplitudes, positions, o, p = d["amplitudes"], d["positions"], d["object"], d["probe"]
    slices, rows, columns = case["slices"], case["rows"], case["columns"]
    shape, n, count = o.shape[1:], rows * columns, len(positions)
    o = o.reshape(slices, -1)
    sampling = WAVELENGTH / 64e-3
    k2 = (_frequency(rows) / sampling)[:, None] ** 2 + (_frequency(columns) / sampling)[None, :] ** 2
    prop = torch.exp(-1j * math.pi * WAVELENGTH * 20.0 * k2)
    energy = (amplitudes.double() ** 2).sum()
    centres = torch.round(positions)
    errors = []
    for _ in range(case["iterations"]):
        sums = _Sums(o.shape[1], slices)
        grad_p, weight_p, error = torch.zeros_like(p), torch.zeros(rows, columns, dtype=torch.float64, device="cuda"), 0.0
        spectrum = torch.fft.fft2(p)
        for b, e in _chunks(count, n, 2 * slices):
            index = _windows(centres[b:e].long(), rows, columns, *shape)
            current = _shifted(spectrum, (positions - centres)[b:e])
            waves, patches = [], []
            for s in range(slices):
                waves.append(current)
                patches.append(o[s][index])
                leaving = current * patches[s]
                if s + 1 < slices:
                    current = torch.fft.ifft2(torch.fft.fft2(leaving) * prop)
            residual, part = _project(torch.fft.fft2(leaving), amplitudes[b:e].double())
            error = error + part
            chi = torch.fft.ifft2(residual)
            for s in range(slices - 1, -1, -1):
                sums.add(s, index, waves[s], chi)
                chi = chi * torch.conj(patches[s])
                if s > 0:
                    chi = torch.fft.ifft2(torch.fft.fft2(chi) * torch.conj(prop))
            grad_p = grad_p + chi.sum(0)
            weight_p = weight_p + (patches[0].real ** 2 + patches[0].imag ** 2).sum(0)
        o = torch.stack([_capped(o[s] + 0.5 * _inverse(sums.weight[s].max()) * torch.view_as_complex(sums.grad[s]))
                         for s in range(slices)])
        p = p + 0.5 * _inverse(weight_p.max()) * grad_p
        errors.append(float(error / energy))
    return o.reshape(slices, *shape), p, np.array(errors)


def _prepared(case, seed):
    cube, origins = _patterns(case, seed)
    count, rows, columns = cube.shape

    def taps(origin, n):
        x = torch.arange(n, dtype=torch.float64, device="cuda") + origin[:, None]
        f = torch.floor(x)
        t = x - f
        if case["shift"] == "bilinear":
            return [(torch.remainder(f.long() + i, n), w) for i, w in ((0, 1 - t), (1, t))]
        return [(torch.remainder(f.long() + i, n), w) for i, w in
                ((-1, (1 - t) ** 3 / 6), (0, (3 * t ** 3 - 6 * t ** 2 + 4) / 6),
                 (1, (-3 * t ** 3 + 3 * t ** 2 + 3 * t + 1) / 6), (2, t ** 3 / 6))]

    values = torch.empty(count, rows, columns, dtype=torch.float64, device="cuda")
    total = clipped = 0.0
    for b, e in _chunks(count, rows * columns):
        v = cube[b:e].double()
        if case["shift"] == "cubicSpline":
            hr, hc = ((4 + 2 * torch.cos(2 * math.pi * _frequency(n))) / 6 for n in (rows, columns))
            v = torch.fft.ifft2(torch.fft.fft2(v) / (hr[:, None] * hc[None, :])).real
        v = sum(w[:, :, None] * torch.gather(v, 1, i[:, :, None].expand(-1, -1, columns))
                for i, w in taps(origins[b:e, 0], rows))
        v = sum(w[:, None, :] * torch.gather(v, 2, i[:, None, :].expand(-1, rows, -1))
                for i, w in taps(origins[b:e, 1], columns))
        total += float(v.sum())
        v = torch.clamp(v, min=0)
        clipped += float(v.sum())
        values[b:e] = torch.sqrt(v)
    return values, total / count, clipped / count


def exact(case, seed):
    kind = case["kind"]
    if kind == "prepare":
        return _prepared(case, seed)
    if kind == "batch":
        return [_reconstructed(c, s)[:3] for c, s in _items(case, seed)]
    if kind == "adjoint":
        loss, grad_object, grad_probe = _reconstructed(case, seed, gradients_only=True)
        return np.array([float(loss)] * 2), grad_object, grad_probe
    if kind == "multislice":
        return _sliced(case, seed)
    o, p, errors, positions = _reconstructed(case, seed)
    if kind == "mixed":
        return o, None, errors  # an eigenvector's phase is free
    if kind == "positions":
        return o, p, errors, positions
    return o, p, errors
