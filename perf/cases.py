"""Performance cases: the work users of rcabeam_b200 run, through its public entry points.

``listed()`` names the standing cases, ``draw(rng)`` gives further cases of the
same ranges.  ``prepare`` builds what a program holds before the call (seeded
inputs, plans), ``run`` makes one pass, ``work`` states the bytes and operations
a pass cannot do without, and ``exact`` restates the result in float64 with
plain torch.

Kinds of case
* ``filtered``   resident filtered-OPW pipeline (``FilteredOpw.run``), both filter
                 domains and every packed storage;
* ``workspace``  ``OpwWorkspace.pack`` + ``reconstruct`` of resident channels;
* ``ensemble``   the NumPy entry points ``beamform_ensemble`` (``signal``) and
                 ``ensemble_pd_from_channels``: host channels in, host maps out;
* ``svd``        ``svd_clutter_filter`` of resident IQ (filtered IQ out);
* ``casorati``   ``temporal_basis`` + ``filtered_power`` of a resident Casorati matrix;
* ``gradient``   ``opw_power_doppler`` forward and backward of a region's loss;
* ``queue``      ``BatchQueue`` replay of an uneven queue of ensembles.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from rcabeam_b200 import beamform_ensemble, ensemble_pd_from_channels
from rcabeam_b200.autograd import DasGeometry, opw_power_doppler
from rcabeam_b200.batching import BatchQueue, Ensemble
from rcabeam_b200.gpu import OpwWorkspace
from rcabeam_b200.gpu_clutter import filtered_power, svd_clutter_filter, temporal_basis
from rcabeam_b200.pipeline import FilteredOpw
from rcabeam_b200.scenes import clutter_casorati
from rcabeam_b200.sim import RCAGeometry

SPEED, RATE, DEMOD = 1540.0, 20e6, 15e6
PRF = 500.0
# How the queue's methods run: per-ensemble grids for OPW, the persistent kernel
# at three CTAs per SM for the others (the autotuner's usual choice).
QUEUE_MODES = {"opw": 0, "xdoppler": 3, "dmas": 3}
# The frame-wise methods' flops per interpolated sample (voxel x element x angle x
# frame): two lerp differences, two lerp FMAs, four FMAs of the rotate-accumulate.
FLOPS_PER_SAMPLE = 14
# Interpolated samples up to which the float64 restatement stays within seconds.
EXACT_SAMPLES = 3.0e11


def listed() -> list[dict]:
    return [
        # A probe-side preview: the smallest acquisition of the test scenes, filtered
        # with the reference's defaults (float32 channels, float64 Gram).
        _das("preview_filtered", "filtered", (256, 64, 5, 16), (32, 64, 32), depth=(3e-3, 15e-3), pitch=0.2e-3,
             storage="float32", precision="complex128", domain="beamformed", rank=3),
        # A notebook user's call: host arrays in, complex IQ back, f-number aperture.
        _das("notebook_iq", "ensemble", (256, 64, 5, 33), (31, 65, 29), depth=(3e-3, 13e-3), pitch=0.2e-3,
             fnumber=1.2, method="opw", signal=True, k=2, storage="float32"),
        # The reference's nonlinear compounding of host channels to a power map.
        _das("host_rc_fmas", "ensemble", (384, 128, 7, 64), (48, 96, 48), method="rc_fmas", signal=False, k=2,
             storage="float32"),
        # Sub-aperture weighting of host channels, odd sizes and a full aperture.
        _das("host_st_sw", "ensemble", (400, 96, 9, 90), (37, 51, 35), pitch=0.15e-3, method="st_sw", signal=False,
             k=3, storage="float32"),
        # Repeated reconstruction on a resident workspace at reference precision: a dense
        # block of the full-size grid (its spacing, its 200-frame ensemble).
        _das("workspace_float32", "workspace", (512, 128, 11, 200), (64, 96, 64), depth=(5e-3, 8e-3), span=0.5,
             storage="float32"),
        # The same with half-size packed channels over the whole aperture, coarser grid.
        _das("workspace_float16", "workspace", (512, 128, 11, 100), (64, 128, 64), storage="float16"),
        # Channel-domain filtering of an odd acquisition before beamforming.
        _das("channel_filtered", "filtered", (300, 96, 9, 75), (40, 70, 36), pitch=0.15e-3, storage="float32",
             precision="complex128", domain="channel", rank=4),
        # The headline workload: full aperture, full grid, split-BF16 tensor-core DAS and Gram.
        _das("filtered_full", "filtered", (512, 128, 11, 200), (128, 256, 128), storage="bf16x2",
             precision="bf16x3", domain="beamformed", rank=3),
        # Clutter filter of beamformed IQ at the default (reference) precision.
        {"name": "svd_filter", "kind": "svd", "rows": 524288, "frames": 200, "rank": 3, "precision": "complex128"},
        # Full-size Casorati matrix: tensor-core Gram, basis and filtered power.
        {"name": "casorati_power", "kind": "casorati", "rows": 4194304, "frames": 400, "rank": 3,
         "precision": "bf16x3"},
        # Calibration by gradient descent: whole-grid power, loss on a 1 mm region.
        _das("calibration_gradient", "gradient", (384, 128, 7, 32), (64, 128, 64), radius=1e-3),
        # A mixed acquisition queue under one CUDA graph.
        {"name": "mixed_queue", "kind": "queue", "samples": 512, "channels": 128, "lateral": 48,
         "items": "opw:96:5:100 dmas:64:7:50 xdoppler:80:5:100 opw:64:11:50 dmas:96:5:33 xdoppler:48:7:200"},
    ]


def draw(rng) -> dict:
    kind = rng.choice(["filtered", "filtered", "workspace", "ensemble", "ensemble", "svd", "casorati", "gradient",
                       "queue"])
    if kind == "svd":
        return {"kind": kind, "rows": _log_int(rng, 20000, 1500000), "frames": rng.randint(16, 256),
                "rank": rng.randint(1, 4), "precision": rng.choice(["complex128", "complex128", "complex64"])}
    if kind == "casorati":
        return {"kind": kind, "rows": _log_int(rng, 100000, 3000000), "frames": 2 * rng.randint(32, 200),
                "rank": rng.randint(2, 4), "precision": rng.choice(["bf16x3", "tf32"])}
    if kind == "queue":
        items = []
        for _ in range(rng.randint(3, 6)):
            items.append(f"{rng.choice(['opw', 'opw', 'xdoppler', 'dmas'])}:{rng.randint(24, 96)}:"
                         f"{rng.choice([3, 5, 7, 11])}:{rng.randint(16, 128)}")
        return {"kind": kind, "samples": rng.randint(300, 512), "channels": rng.choice([64, 96, 128]),
                "lateral": rng.randint(24, 48), "items": " ".join(items)}
    nc = rng.choice([48, 64, 96, 128])
    channels = (rng.randint(256, 512), nc, rng.choice([3, 5, 7, 9, 11]), _log_int(rng, 12, 200))
    pitch = 14e-3 / nc
    fnumber = rng.choice([0.0, 0.0, 1.0, 1.5])
    budget = {"filtered": 1.5e11, "workspace": 1.5e11, "ensemble": 3e10, "gradient": 3e10}[kind]
    grid = _draw_grid(rng, channels, budget)
    if kind == "gradient":
        return _das(None, kind, channels[:3] + (min(channels[3], 64),), grid, pitch=pitch, fnumber=fnumber,
                    radius=rng.uniform(0.6e-3, 1.2e-3))
    if kind == "workspace":
        return _das(None, kind, channels, grid, pitch=pitch, fnumber=fnumber, span=rng.choice([0.5, 1.0]),
                    storage=rng.choice(["float32", "float32", "float16"]))
    if kind == "filtered":
        storage = rng.choice(["float32", "bf16x2"])
        if storage == "bf16x2":
            channels = channels[:3] + (4 * max(4, channels[3] // 4),)
        precision = rng.choice(["complex128", "bf16x3"]) if channels[3] % 2 == 0 else "complex128"
        return _das(None, kind, channels, grid, pitch=pitch, fnumber=fnumber, storage=storage, precision=precision,
                    domain=rng.choice(["beamformed", "beamformed", "channel"]), rank=rng.randint(3, 4))
    method = rng.choice(["opw", "opw", "xdoppler", "rc_fmas", "dmas", "st_sw"])
    signal = method in ("opw", "xdoppler", "rc_fmas") and rng.random() < 0.3
    return _das(None, kind, channels, grid, pitch=pitch, fnumber=fnumber, method=method, signal=signal,
                k=rng.randint(2, 3), storage="float32")


def prepare(case: dict, seed: int):
    kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind in ("svd", "casorati"):
        return {"case": case, "iq": _casorati(case, gen)}
    if kind == "queue":
        ensembles = []
        for item, (method, shape, grid, geom, angles, t_start) in enumerate(_queue_items(case)):
            packed = [c.permute(1, 2, 0, 3).contiguous() for c in _channels(shape, geom, angles, t_start, gen)]
            e = Ensemble(packed[0], packed[1], shape, grid, geom, angles, t_start, method)
            e.build(packed[0].device)
            ensembles.append(e)
        queue = BatchQueue(ensembles, ctas_per_sm=QUEUE_MODES)
        queue.capture()
        return {"case": case, "queue": queue}
    shape, grid, geom, angles, t_start = _acquisition(case)
    rc, cr = _channels(shape, geom, angles, t_start, gen)
    state = {"case": case, "rc": rc, "cr": cr, "angles": angles, "t_start": t_start, "grid": grid, "geom": geom}
    if kind == "filtered":
        state["plan"] = FilteredOpw(shape, angles, t_start, grid, geom, rank_start=case["rank"],
                                    precision=case["precision"], iq_storage=case["storage"], domain=case["domain"])
    elif kind == "workspace":
        state["plan"] = OpwWorkspace(shape, angles, t_start, grid, geom, iq_storage=case["storage"])
    elif kind == "ensemble":
        state["rc"], state["cr"] = rc.cpu().numpy(), cr.cpu().numpy()
    elif kind == "gradient":
        state["geometry"] = DasGeometry.build(grid, geom, angles, t_start)
        state["offsets"] = _offsets(case, seed)
        state["roi"] = _region(case, _scan(grid))
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "filtered":
        return state["plan"].run(state["rc"], state["cr"])
    if kind == "workspace":
        plan = state["plan"]
        plan.pack(state["rc"], state["cr"])
        iq = plan.reconstruct()
        return iq, plan.power
    if kind == "ensemble":
        args = (state["rc"], state["cr"], state["angles"], state["t_start"], state["grid"], state["geom"])
        if case["signal"]:
            return beamform_ensemble(*args, method=case["method"], iq_storage=case["storage"])
        return ensemble_pd_from_channels(*args, method=case["method"], k=case["k"], iq_storage=case["storage"])
    if kind == "svd":
        return svd_clutter_filter(state["iq"], rank_start=case["rank"], precision=case["precision"])
    if kind == "casorati":
        values, basis = temporal_basis(state["iq"], precision=case["precision"])
        return values, filtered_power(state["iq"], basis, rank_start=case["rank"])
    if kind == "gradient":
        rc, cr = state["rc"].detach().requires_grad_(), state["cr"].detach().requires_grad_()
        offsets = state["offsets"].detach().requires_grad_()
        speed = torch.tensor(1523.0, dtype=torch.float64, device=rc.device, requires_grad=True)
        power = opw_power_doppler(rc, cr, offsets, speed, state["geometry"])
        (power * state["roi"]).sum().backward()
        return power.detach(), rc.grad, cr.grad, offsets.grad, speed.grad
    queue = state["queue"]
    queue.run()
    return [e.power() for e in queue.ensembles]


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("svd", "casorati"):
        rows, t, k = case["rows"], case["frames"], case["rank"]
        out = 8 * rows * t if kind == "svd" else 8 * rows
        # Upper triangle of the Gram, k coordinates and the k-term residual.
        return {"bytes": 8 * rows * t + out, "flops": rows * (4 * t * t + 16 * k * t)}
    if kind == "queue":
        total_bytes = total_flops = 0
        for _, shape, grid, *_ in _queue_items(case):
            voxels = math.prod(len(axis) for axis in grid)
            total_bytes += 16 * math.prod(shape) + 4 * voxels
            total_flops += FLOPS_PER_SAMPLE * voxels * 2 * math.prod(shape[1:])
        return {"bytes": total_bytes, "flops": total_flops}
    shape, grid, *_ = _acquisition(case)
    voxels, frames = math.prod(len(axis) for axis in grid), shape[3]
    channels = 16 * math.prod(shape)
    flops = FLOPS_PER_SAMPLE * voxels * 2 * math.prod(shape[1:])
    if kind == "workspace":
        return {"bytes": channels + 8 * voxels * frames + 4 * voxels, "flops": flops}
    if kind == "ensemble":
        return {"bytes": channels + (8 * voxels * frames if case["signal"] else 4 * voxels), "flops": flops}
    if kind == "gradient":
        listed_voxels = int(_region(case, _scan(grid, "cpu")).sum())
        return {"bytes": 2 * channels + 8 * voxels,
                "flops": flops + 4 * FLOPS_PER_SAMPLE * listed_voxels * 2 * math.prod(shape[1:])}
    rows = voxels if case["domain"] == "beamformed" else 2 * math.prod(shape[:3])
    return {"bytes": channels + 8 * voxels, "flops": flops + rows * (4 * frames**2 + 16 * case["rank"] * frames)}


def exact(case: dict, seed: int):
    kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    if kind in ("svd", "casorati"):
        iq = _casorati(case, gen)
        values, discarded = _exact_basis([iq], case["rank"])
        if kind == "svd":
            return _exact_residual(iq, discarded)
        parts = iq.split(1 << 19)
        return values, torch.cat([_exact_residual(p, discarded).abs().square().mean(-1) for p in parts])
    if kind == "queue":
        out = []
        for method, shape, grid, geom, angles, t_start in _queue_items(case):
            rc, cr = _channels(shape, geom, angles, t_start, gen)
            out.append(_exact_power(method, rc, cr, grid, geom, angles, t_start))
        return out
    shape, grid, geom, angles, t_start = _acquisition(case)
    if math.prod(len(axis) for axis in grid) * 2 * math.prod(shape[1:]) > EXACT_SAMPLES:
        return None
    rc, cr = _channels(shape, geom, angles, t_start, gen)
    args = (grid, geom, angles, t_start)
    dims = tuple(len(axis) for axis in grid)
    if kind == "workspace":
        iq = _exact_opw(rc, cr, *args)
        return iq.reshape(*dims, -1), iq.abs().square().mean(-1).reshape(dims)
    if kind == "ensemble":
        if case["signal"]:
            iq = _exact_signal(case["method"], rc, cr, *args)
            return iq.reshape(*dims, -1).cpu().numpy()
        return _exact_power(case["method"], rc, cr, *args, k=case["k"]).reshape(dims).cpu().numpy()
    if kind == "gradient":
        return _exact_gradient(case, seed, rc, cr, *args)
    if case["domain"] == "channel":
        _, discarded = _exact_basis([rc, cr], case["rank"])
        rc, cr = (_exact_residual(c, discarded).reshape(shape) for c in (rc, cr))
        return _exact_opw(rc, cr, *args).abs().square().mean(-1).reshape(dims)
    iq = _exact_opw(rc, cr, *args)
    _, discarded = _exact_basis([iq], case["rank"])
    return _exact_residual(iq, discarded).abs().square().mean(-1).reshape(dims)


# ------------------------------------------------------------------ inputs --
def _das(name, kind, channels, grid, *, depth=(4e-3, 12e-3), pitch=0.11e-3, fnumber=0.0, span=1.0, **fields) -> dict:
    """One acquisition: channels (samples, elements, angles, frames) on an (x, z, y) grid that
    spans ``span`` of the aperture; ``fnumber`` 0 is the full aperture."""
    case = {} if name is None else {"name": name}
    case.update(kind=kind, samples=channels[0], channels=channels[1], angles=channels[2], frames=channels[3],
                nx=grid[0], nz=grid[1], ny=grid[2], z0=depth[0], z1=depth[1], pitch=pitch, fnumber=fnumber,
                span=span)
    case.update(fields)
    return case


def _log_int(rng, low: int, high: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _draw_grid(rng, channels, budget: float) -> tuple[int, int, int]:
    """A grid of 1/8 to all of the voxels that ``budget`` interpolated samples allow."""
    voxels = budget / (2 * math.prod(channels[1:])) * math.exp(rng.uniform(math.log(1 / 8), 0.0))
    side = min(max(voxels, 4096.0), 600000.0) ** (1 / 3)
    nx, ny = max(8, int(side * rng.uniform(0.6, 1.0))), max(8, int(side * rng.uniform(0.6, 1.0)))
    return nx, max(8, int(side**3 / (nx * ny))), ny


def _geometry(elements: int, pitch: float, fnumber: float) -> RCAGeometry:
    el = (np.arange(elements) - (elements - 1) / 2) * pitch
    return RCAGeometry(el, el, c=SPEED, fs=RATE, f_demod=DEMOD, fnumber=fnumber or None)


def _start(z0: float) -> float:
    """Sampling starts half a microsecond before the echo of the shallowest depth."""
    return 2 * z0 / SPEED - 0.5e-6


def _acquisition(case):
    shape = (case["samples"], case["channels"], case["angles"], case["frames"])
    geom = _geometry(case["channels"], case["pitch"], case["fnumber"])
    angles = np.deg2rad(np.linspace(-10, 10, case["angles"]))
    half = (case["channels"] - 1) / 2 * case["pitch"] * case["span"]
    grid = (np.linspace(-half, half, case["nx"]), np.linspace(case["z0"], case["z1"], case["nz"]),
            np.linspace(-half, half, case["ny"]))
    return shape, grid, geom, angles, _start(case["z0"])


def _queue_items(case):
    """(method, shape, grid, geometry, angles, start) of each ``method:depth:angles:frames`` item."""
    pitch = 14e-3 / case["channels"]
    geom = _geometry(case["channels"], pitch, 0.0)
    half = 14e-3 / 2 * case["lateral"] / 128
    for item in case["items"].split():
        method, depth, angles, frames = item.split(":")
        shape = (case["samples"], case["channels"], int(angles), int(frames))
        lateral = np.linspace(-half, half, case["lateral"])
        grid = (lateral, 4e-3 + 8e-3 / 255 * np.arange(int(depth)), lateral)
        yield method, shape, grid, geom, np.deg2rad(np.linspace(-10, 10, int(angles))), _start(4e-3)


def _channels(shape, geom: RCAGeometry, angles, t_start: float, gen: torch.Generator):
    """RC and CR channels ``(samples, elements, angles, frames)`` of a seeded flow scene: point
    scatterers of slowly moving tissue (three temporal modes), four groups of blood
    scatterers 40 dB lower with their own Doppler, white noise at -50 dB."""
    ns, nc, na, nt = shape
    dev = gen.device
    rand = lambda *s: torch.rand(*s, generator=gen, device=dev, dtype=torch.float64)  # noqa: E731
    frame = torch.arange(nt, device=dev, dtype=torch.float64)
    tissue = 2 * math.pi * (2 * 1e-3 * DEMOD / SPEED) / PRF
    groups = []  # (scatterers, amplitude, temporal mode)
    for m, level in enumerate((0.0, -6.0, -12.0)):
        mode = torch.polar(torch.cos(math.pi * m * (frame + 0.5) / nt), tissue * frame)
        groups.append((16, 10 ** (level / 20), mode))
    for speed in (10e-3, 16e-3, 22e-3, 28e-3):
        doppler = 2 * math.pi * (2 * speed * DEMOD / SPEED) / PRF
        groups.append((6, 0.01, torch.polar(torch.ones_like(frame), doppler * frame)))
    half = float(np.abs(geom.x_el).max())
    far = (t_start + ns / RATE) * SPEED / 2
    near = (t_start + 0.5e-6) * SPEED / 2
    scene = []
    for count, level, mode in groups:
        x, z, y = (2 * rand(count) - 1) * half, near + rand(count) * (far - near), (2 * rand(count) - 1) * half
        amp = torch.polar(level * (0.5 + rand(count)), 2 * math.pi * rand(count))
        scene.append((x, z, y, amp, mode.to(torch.complex64)))
    ang = torch.as_tensor(np.asarray(angles, np.float32), device=dev).double()
    t = t_start + torch.arange(ns, device=dev, dtype=torch.float64)[:, None, None] / RATE
    out = []
    for config, el in enumerate((geom.x_el, geom.y_el)):
        e = torch.as_tensor(np.asarray(el, np.float32), device=dev).double()
        data = torch.complex(*(torch.randn(shape, generator=gen, device=dev) for _ in range(2)))
        fields, level = [], 0.0
        for x, z, y, amp, mode in scene:
            field = torch.zeros((ns, nc, na), dtype=torch.complex64, device=dev)
            rx, tx = (y, x) if config else (x, y)
            for i in range(len(x)):
                tau = (((z[i] * torch.cos(ang) + tx[i] * torch.sin(ang)) / SPEED)[None, None, :]
                       + (torch.sqrt(z[i] ** 2 + (rx[i] - e) ** 2) / SPEED)[None, :, None])
                envelope = torch.exp(-(((t - tau) / 0.15e-6) ** 2)).float()
                field += envelope * (amp[i] * torch.polar(torch.ones_like(tau), -2 * math.pi * DEMOD * tau)).to(
                    torch.complex64)
            fields.append((field, mode))
            level += float((field.abs() ** 2).double().mean())
        data *= math.sqrt(level * 1e-5 / 2)
        for field, mode in fields:
            data += field[..., None] * mode
        out.append(data)
    return out


def _casorati(case, gen: torch.Generator) -> torch.Tensor:
    return clutter_casorati(case["rows"], case["frames"], generator=gen, device=gen.device)


def _offsets(case, seed: int) -> torch.Tensor:
    noise = np.random.default_rng(seed).normal(scale=5e-9, size=(2, case["channels"]))
    return torch.as_tensor(noise, device="cuda")


def _region(case, scan: torch.Tensor) -> torch.Tensor:
    """Loss weights on the (x, z, y) grid: one inside a sphere about the grid's centre."""
    centre = scan.new_tensor([0.1e-3, 0.5 * (case["z0"] + case["z1"]), -0.1e-3])
    inside = (scan - centre).square().sum(-1) <= case["radius"] ** 2
    return inside.double().reshape(case["nx"], case["nz"], case["ny"])


# -------------------------------------------------- float64 restatement --
def _scan(grid, device="cuda") -> torch.Tensor:
    """Voxel coordinates (x, z, y) in float64 of the float32 grid, x-major and y innermost."""
    axes = [torch.as_tensor(np.asarray(a, np.float32), device=device).double() for a in grid]
    return torch.cartesian_prod(*axes)


def _exact_samples(data, scan, el, angles, t_start, geom, config, *, speed=None, offsets=None):
    """Yields (channel, angle, delay, rows, next rows, weights, phase) of one aperture."""
    ns, nc, na, _ = data.shape
    c = geom.c if speed is None else speed
    f64 = lambda a: torch.as_tensor(np.asarray(a, np.float32), device=data.device).double()  # noqa: E731
    el, angles, start = f64(el), f64(angles), float(np.float32(t_start))
    x, z, y = scan.unbind(1)
    rx, tx = (y, x) if config else (x, y)
    for ch in range(nc):
        distance = rx - el[ch]
        receive = torch.sqrt(z * z + distance * distance) / c
        if offsets is not None:
            receive = receive + offsets[config, ch]
        for a in range(na):
            tau = (z * torch.cos(angles[a]) + tx * torch.sin(angles[a])) / c + receive
            sample = (tau - start) * geom.fs
            valid = (sample >= 0) & (sample <= ns - 1)
            if geom.fnumber is not None:
                valid &= distance.abs() <= z / (2 * float(np.float32(geom.fnumber)))
            sample = sample.clamp(0, ns - 1)
            row = sample.floor()
            weight = sample - row
            row = row.long()
            phase = torch.polar(valid.double(), 2 * math.pi * torch.remainder(geom.f_demod * tau, 1.0))
            yield ch, a, tau, row, (row + 1).clamp(max=ns - 1), weight, phase


def _exact_terms(data, scan, el, angles, t_start, geom, config, **extra):
    """Yields (channel, angle, (voxels, frames) complex128 term) of one aperture's delay-and-sum."""
    for ch, a, _, row, nxt, weight, phase in _exact_samples(data, scan, el, angles, t_start, geom, config, **extra):
        slab = data[:, ch, a].to(torch.complex128)
        term = slab[row] * (phase * (1 - weight))[:, None]
        yield ch, a, term.addcmul_(slab[nxt], (phase * weight)[:, None])


def _blocks(grid, frames: int, planes: int = 1):
    return _scan(grid).split(max(1, (1 << 26) // (frames * planes)))


def _exact_opw(rc, cr, grid, geom, angles, t_start, **extra) -> torch.Tensor:
    out = []
    for scan in _blocks(grid, rc.shape[3]):
        acc = torch.zeros((len(scan), rc.shape[3]), dtype=torch.complex128, device=rc.device)
        for config, (data, el) in enumerate(((rc, geom.x_el), (cr, geom.y_el))):
            for _, _, term in _exact_terms(data, scan, el, angles, t_start, geom, config, **extra):
                acc += term
        out.append(acc)
    return torch.cat(out)


def _signed_sqrt(x: torch.Tensor) -> torch.Tensor:
    magnitude = x.abs()
    return torch.where(magnitude > 0, x / magnitude.clamp(min=1e-300).sqrt(), torch.zeros_like(x))


def _exact_signal(method, rc, cr, grid, geom, angles, t_start) -> torch.Tensor:
    """Slow-time signal (voxels, frames) of OPW, XDoppler or RC-FMAS."""
    if method == "opw":
        return _exact_opw(rc, cr, grid, geom, angles, t_start)
    out = []
    for scan in _blocks(grid, rc.shape[3], rc.shape[2]):
        r, q = (_exact_angles(scan, data, el, angles, t_start, geom, config)[0]
                for config, (data, el) in enumerate(((rc, geom.x_el), (cr, geom.y_el))))
        out.append(_signed_sqrt(r).sum(0) * _signed_sqrt(q).sum(0) if method == "rc_fmas"
                   else r.sum(0) * q.sum(0).conj())
    return torch.cat(out)


def _exact_angles(scan, data, el, angles, t_start, geom, config):
    """Per-angle sums (angles, voxels, frames), and the signed-root and magnitude sums of the
    per-channel sums with the count of channels inside the aperture."""
    _, nc, na, nt = data.shape
    per_angle = torch.zeros((na, len(scan), nt), dtype=torch.complex128, device=data.device)
    root = torch.zeros_like(per_angle[0])
    magnitude = torch.zeros(root.shape, dtype=torch.float64, device=data.device)
    channel = None
    for _, a, term in _exact_terms(data, scan, el, angles, t_start, geom, config):
        per_angle[a] += term
        channel = term.clone() if a == 0 else channel.add_(term)
        if a == na - 1:
            root += _signed_sqrt(channel)
            magnitude += channel.abs()
    coords = scan[:, 2 if config else 0, None] - torch.as_tensor(np.asarray(el, np.float32),
                                                                 device=scan.device).double()
    limit = math.inf if geom.fnumber is None else scan[:, 1:2] / (2 * float(np.float32(geom.fnumber)))
    return per_angle, root, magnitude, (coords.abs() <= limit).sum(1).double()


def _exact_power(method, rc, cr, grid, geom, angles, t_start, k: int = 2) -> torch.Tensor:
    if method in ("opw", "rc_fmas"):
        return _exact_signal(method, rc, cr, grid, geom, angles, t_start).abs().square().mean(-1)
    if method == "xdoppler":
        return _exact_signal(method, rc, cr, grid, geom, angles, t_start).mean(-1).abs()
    power, weights = [], []
    for scan in _blocks(grid, rc.shape[3], 2 * rc.shape[2]):
        (r, root_r, mag_r, n_r), (q, root_q, mag_q, n_q) = (
            _exact_angles(scan, data, el, angles, t_start, geom, config)
            for config, (data, el) in enumerate(((rc, geom.x_el), (cr, geom.y_el))))
        if method == "dmas":
            power.append(_exact_dmas(r, q, root_r + root_q, mag_r + mag_q, n_r + n_q))
        else:
            power.append((r.sum(0) * q.sum(0).conj()).mean(-1).abs())
            weights.append(_exact_pairs(r, q, k))
    power = torch.cat(power)
    if method == "st_sw":
        weight = torch.cat(weights)
        power = power * (weight / weight.max())
    return power


def _spread(x: torch.Tensor):
    mean = x.mean(0)
    return mean, (x - mean).abs().square().mean(0)


def _ratio(num: torch.Tensor, den: torch.Tensor) -> torch.Tensor:
    return torch.where(den > 0, num / torch.where(den > 0, den, torch.ones_like(den)), torch.zeros_like(num))


def _exact_dmas(r, q, root, magnitude, active) -> torch.Tensor:
    response = root.abs().square() - magnitude
    coherence = _ratio(_ratio(response.clamp(min=0), magnitude), active[:, None].expand_as(magnitude))
    (mr, vr), (mq, vq) = _spread(r), _spread(q)
    num = (mr * mq.conj()).abs()
    angular = _ratio(num, mr.abs().square() + mq.abs().square() + (vr + vq) / 2 - num)
    return (response * coherence * angular).mean(-1)


def _exact_pairs(r, q, k: int) -> torch.Tensor:
    """Raw sub-aperture weights: normalized pair sum of the k x k subset correlation series."""
    sr, sq = [_spread(r[i::k]) for i in range(k)], [_spread(q[i::k]) for i in range(k)]
    series = {}
    for i, (mr, vr) in enumerate(sr):
        for j, (mq, vq) in enumerate(sq):
            num = mr * mq.conj()
            den = mr.abs().square() + mq.abs().square() + (vr + vq) / 2 - num.abs()
            value = _ratio(num, den)
            series[i, j] = _ratio(value, value.abs().square().sum(-1, keepdim=True).sqrt().expand_as(den))
    total = torch.zeros(r.shape[1], dtype=torch.complex128, device=r.device)
    for (i1, j1), first in series.items():
        for (i2, j2), second in series.items():
            if i1 < i2 and j1 != j2:
                total += (first * second.conj()).sum(-1)
    return total.abs()


def _exact_basis(arrays, rank: int):
    """Singular values and the ``rank`` leading temporal vectors of the stacked Casorati rows."""
    frames = arrays[0].shape[-1]
    gram = torch.zeros((frames, frames), dtype=torch.complex128, device=arrays[0].device)
    for a in arrays:
        for part in a.reshape(-1, frames).split(1 << 19):
            part = part.to(torch.complex128)
            gram += part.mH @ part
    lam, vectors = torch.linalg.eigh(gram)
    return lam.flip(0).clamp(min=0).sqrt(), vectors.flip(1)[:, :rank]


def _exact_residual(iq, discarded) -> torch.Tensor:
    rows = iq.reshape(-1, iq.shape[-1]).to(torch.complex128)
    return rows.addmm(rows @ discarded, discarded.mH, alpha=-1)


def _exact_gradient(case, seed, rc, cr, grid, geom, angles, t_start):
    """Power of the whole grid and the gradients of the region's summed power."""
    nt = rc.shape[3]
    scan = _scan(grid)
    roi = _region(case, scan)
    extra = {"speed": 1523.0, "offsets": _offsets(case, seed)}
    iq = _exact_opw(rc, cr, grid, geom, angles, t_start, **extra)
    inside = roi.flatten().nonzero().flatten()
    upstream = (2.0 / nt) * iq[inside]
    grads, d_offsets, d_speed = [], torch.zeros_like(extra["offsets"]), torch.zeros((), dtype=torch.float64,
                                                                                    device=rc.device)
    for config, (data, el) in enumerate(((rc, geom.x_el), (cr, geom.y_el))):
        grad = torch.zeros((*data.shape[1:3], data.shape[0], nt), dtype=torch.complex128, device=rc.device)
        for ch, a, tau, row, nxt, weight, phase in _exact_samples(data, scan[inside], el, angles, t_start, geom,
                                                                  config, **extra):
            slab = data[:, ch, a].to(torch.complex128)
            back = upstream * phase.conj()[:, None]
            grad[ch, a].index_add_(0, row, back * (1 - weight)[:, None])
            grad[ch, a].index_add_(0, nxt, back * weight[:, None])
            step = (slab[nxt] - slab[row]) * phase[:, None]
            term = (slab[row] * (1 - weight)[:, None] + slab[nxt] * weight[:, None]) * phase[:, None]
            d_tau = (upstream.conj() * (geom.fs * step + 2j * math.pi * geom.f_demod * term)).real.sum(1)
            d_offsets[config, ch] += d_tau.sum()
            d_speed -= (d_tau * (tau - extra["offsets"][config, ch])).sum() / extra["speed"]
        grads.append(grad.permute(2, 0, 1, 3))
    power = iq.abs().square().mean(-1).reshape(roi.shape)
    return power, grads[0], grads[1], d_offsets, d_speed
