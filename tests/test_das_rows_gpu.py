"""Edges of the staged delay-and-sum kernel against the float64 oracle: item and
thread splits of the frames, odd frame counts and unaligned buffers (bulk copies),
windows longer than a ring stage, tiles that fall apart, many angles, apertures
no voxel of a tile reaches.  Bars as in test_das_gpu.py (IQ 1e-5, products of
sums 1e-4)."""

from __future__ import annotations

import threading

import numpy as np
import pytest
import torch

from oracle import methods
from rcabeam_b200 import _cuda_impl, _lib, batching
from rcabeam_b200.sim import RCAGeometry
from tests._cases import rel_l2

pytestmark = pytest.mark.gpu
FS, FD, C = 20e6, 5e6, 1540.0


@pytest.fixture(autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")
    yield
    assert _lib.device_error() == 0


def _voxels(kind: str, nv: int, rng) -> np.ndarray:
    """Positions (x, z, y): within a few sample rows, over the whole window, or in two distant clusters."""
    span = {"dense": 0.2e-3, "coarse": 5e-3, "apart": 0.2e-3}[kind]
    scan = rng.uniform([-1e-3, 3e-3, -1e-3], [1e-3, 3e-3 + span, 1e-3], (nv, 3))
    if kind == "dense":
        scan[:, ::2] *= 0.1
    if kind == "apart":
        scan[nv // 2:, 1] += 5e-3
    return scan.astype(np.float32)


def _reconstruct(rc, cr, scan, xe, ye, angles, starts, fn, method, shift, c=C, fs=FS, fd=FD,
                 k=2):
    ns, nc, na, nt = rc.shape
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    packed = []
    for src in (rc, cr):  # packed (c, a, s, t), `shift` samples past a 16-byte boundary
        buf = torch.zeros(rc.size + 2, dtype=torch.complex64, device="cuda")
        dst = buf[shift:shift + rc.size]
        dst.copy_(dev(src.transpose(1, 2, 0, 3)).reshape(-1))
        packed.append(dst)
    nv = len(scan)
    pd = torch.empty((nv, 2), dtype=torch.float32, device="cuda")
    planes = 2 if method == 5 else 1
    signal = torch.full((nv * planes, nt), float("nan"), dtype=torch.complex64, device="cuda")
    weights = series = None
    if method == 4:
        weights, signal = torch.empty(nv, dtype=torch.float32, device="cuda"), None
        series = torch.empty(nv * k * k * nt, dtype=torch.complex64, device="cuda")
    work = torch.empty(_cuda_impl.workspace_bytes(nv, nc, na), dtype=torch.uint8, device="cuda")
    t = [dev(a) for a in (scan, xe, ye, angles, starts)]
    _lib.call("rcabeam_ensemble_device", packed[0].data_ptr(), packed[1].data_ptr(), *(a.data_ptr() for a in t),
              pd.data_ptr(), *(None if a is None else a.data_ptr() for a in (signal, weights, series)), work.data_ptr(),
              ns, nc, na, nt, nv, c, fs, fd, -1.0 if fn is None else fn, method, k)
    if method == 4:
        return pd[:, 0].cpu().numpy(), weights.cpu().numpy()
    return pd[:, 0].cpu().numpy(), signal.cpu().numpy().reshape(nv, planes, nt)


@pytest.mark.parametrize("frames,kind,nv,na,fn,shift", [
    (1, "dense", 127, 3, None, 0), (16, "coarse", 129, 5, None, 0), (17, "coarse", 300, 5, 1.0, 1),
    (26, "dense", 128, 4, 1.0, 1), (33, "apart", 257, 3, None, 0), (48, "coarse", 130, 2, 1.0, 0),
    (49, "dense", 150, 3, None, 1), (64, "apart", 200, 3, None, 0), (65, "dense", 129, 3, 1.0, 0),
    (104, "coarse", 140, 2, None, 0), (105, "coarse", 131, 2, 1.0, 1), (106, "dense", 129, 3, None, 0),
    (209, "apart", 130, 2, None, 0), (6, "coarse", 140, 180, None, 0),
])
def test_staged_splits_match_oracle(frames, kind, nv, na, fn, shift):
    rng = np.random.default_rng(frames + nv)
    ns, nc = 200, 7
    f64 = lambda a: np.asarray(a, np.float32).astype(np.float64)  # noqa: E731
    scan = _voxels(kind, nv, rng)
    xe = np.linspace(-4e-3, 4e-3, nc).astype(np.float32)
    ye = np.linspace(-3.9e-3, 4.1e-3, nc).astype(np.float32)
    angles = np.linspace(-0.17, 0.16, na).astype(np.float32)
    starts = np.full(na, 2 * 3e-3 / C - 0.4e-6, np.float32)
    shape = (ns, nc, na, frames)
    rc, cr = ((rng.normal(size=shape) + 1j * rng.normal(size=shape)).astype(np.complex64) for _ in range(2))
    geom = (f64(scan), f64(xe), f64(ye), f64(angles), f64(starts), C, FS, FD, fn)
    chan_r, ang_r, n_r = methods.aperture_terms(rc, geom[0], geom[1], *geom[3:], "RC")
    chan_q, ang_q, n_q = methods.aperture_terms(cr, geom[0], geom[2], *geom[3:], "CR")
    r, q = ang_r.sum(axis=1), ang_q.sum(axis=1)
    run = lambda method: _reconstruct(rc, cr, scan, xe, ye, angles, starts, fn, method, shift)  # noqa: E731
    pd, iq = run(0)
    assert rel_l2(iq[:, 0], r + q) <= 1e-5
    assert rel_l2(pd, np.mean(np.abs(r + q) ** 2, axis=-1)) <= 1e-5
    _, iq = run(5)
    assert rel_l2(iq, np.stack((r, q), axis=1)) <= 1e-5
    if na > 8:
        return
    pd, _ = run(1)
    assert rel_l2(pd, np.abs(np.mean(r * q.conj(), axis=-1))) <= 1e-4
    fmas = methods.signed_sqrt(ang_r).sum(axis=1) * methods.signed_sqrt(ang_q).sum(axis=1)
    pd, signal = run(2)
    assert rel_l2(signal[:, 0], fmas) <= 1e-4
    assert rel_l2(pd, np.mean(np.abs(fmas) ** 2, axis=-1)) <= 1e-4
    pd, _ = run(3)
    assert rel_l2(pd, methods.dmas_ccf_acf_power(rc, cr, *geom)) <= 1e-4


@pytest.mark.parametrize("method,k", [(2, 2), (3, 2), (4, 2), (4, 3), (4, 4)])
@pytest.mark.parametrize("frames,kind,nv,na,fn,shift", [
    (1, "dense", 127, 4, None, 0), (17, "coarse", 300, 5, 1.0, 1), (26, "dense", 1, 4, 1.0, 1),
    (33, "apart", 257, 35, None, 0), (48, "coarse", 130, 5, 1.0, 0), (49, "dense", 150, 4, None, 1),
    (97, "coarse", 129, 6, None, 0),
])
def test_nonlinear_routes_agree(method, k, frames, kind, nv, na, fn, shift):
    """A few voxels (a warp each) and the same voxels repeated until the call takes the
    staged kernel, on tiles of one voxel's repetitions and on mixed ones (1e-4: products of sums)."""
    rng = np.random.default_rng(frames + nv)
    ns, nc = 200, 37  # more channels than a warp has lanes, angles too with 35
    scan = _voxels(kind, nv, rng)
    xe = np.linspace(-4e-3, 4e-3, nc).astype(np.float32)
    angles = np.linspace(-0.17, 0.16, na).astype(np.float32)
    starts = np.full(na, 2 * 3e-3 / C - 0.4e-6, np.float32)
    shape = (ns, nc, na, frames)
    rc, cr = ((rng.normal(size=shape) + 1j * rng.normal(size=shape)).astype(np.complex64) for _ in range(2))
    repeats = 16384 // (nv * -(-frames // 32)) + 1
    args = (xe, xe + np.float32(1e-4), angles, starts, fn, method, shift)
    pd, extra = _reconstruct(rc, cr, scan, *args, k=k)
    pd_staged, extra_staged = _reconstruct(rc, cr, np.tile(scan, (repeats, 1)), *args, k=k)
    assert np.abs(pd).max() > 0
    for copy in (slice(0, nv), slice(len(pd_staged) - nv, None)):
        assert rel_l2(pd_staged[copy], pd) <= 1e-4
        assert rel_l2(extra_staged[copy], extra) <= 1e-4


@pytest.mark.parametrize("method,specs", [
    ("xdoppler", [(50, 3), (16, 48), (64, 2)]),  # a long angle table beside wide stages: they shrink
    ("dmas", [(48, 2), (20, 9), (7, 40)]),       # items with two and with three builder warps
])
def test_queue_of_uneven_layouts(method, specs):
    """Ensembles whose own rings differ share one launch (1e-5 as in test_batch_gpu.py)."""
    rng = np.random.default_rng(len(specs))
    ns, nc = 160, 8
    el = (np.arange(nc) - (nc - 1) / 2) * 0.2e-3
    geom = RCAGeometry(el, el, c=C, fs=FS, f_demod=FD, fnumber=None)
    ensembles = []
    for frames, na in specs:
        shape = (ns, nc, na, frames)
        packed = [torch.from_numpy((rng.normal(size=shape) + 1j * rng.normal(size=shape)).astype(np.complex64))
                  .permute(1, 2, 0, 3).contiguous().cuda() for _ in range(2)]
        grid = (np.linspace(-1.2e-3, 1.2e-3, 9), np.linspace(3e-3, 6e-3, 13), np.linspace(-1e-3, 1e-3, 7))
        e = batching.Ensemble(packed[0], packed[1], shape, grid, geom, np.deg2rad(np.linspace(-8, 8, na)), 3e-6, method)
        e.build(torch.device("cuda"))
        ensembles.append(e)
    batching.sequential(ensembles)
    want = [e.power().cpu().numpy().copy() for e in ensembles]
    batching.BatchQueue(ensembles, ctas_per_sm=1).run()
    torch.cuda.synchronize()
    for e, w in zip(ensembles, want):
        assert np.abs(w).max() > 0
        assert rel_l2(e.power().cpu().numpy(), w) <= 1e-5


@pytest.mark.parametrize("method,frames", [("opw", (100, 16)), ("xdoppler", (64, 16))])
def test_queue_of_long_windows(method, frames):
    """A step's window of more than 256 sample rows, 32 boxes, beside an ensemble whose
    ring gives the short one far wider stages (1e-5 as in test_batch_gpu.py)."""
    rng = np.random.default_rng(frames[0])
    ns, nc, na = 800, 6, 5
    el = (np.arange(nc) - (nc - 1) / 2) * 0.2e-3
    geom = RCAGeometry(el, el, c=C, fs=FS, f_demod=FD, fnumber=None)
    grid = (np.linspace(-1e-3, 1e-3, 3), np.linspace(3e-3, 30e-3, 20), np.linspace(-1e-3, 1e-3, 2))  # one tile
    ensembles = []
    for nt in frames:
        packed = [torch.from_numpy((rng.normal(size=(nc, na, ns, nt)) + 1j * rng.normal(size=(nc, na, ns, nt)))
                                   .astype(np.complex64)).cuda() for _ in range(2)]
        e = batching.Ensemble(packed[0], packed[1], (ns, nc, na, nt), grid, geom, np.deg2rad(np.linspace(-8, 8, na)),
                              3e-6, method)
        e.build(torch.device("cuda"))
        ensembles.append(e)
    batching.sequential(ensembles)
    want = [e.power().cpu().numpy().copy() for e in ensembles]
    batching.BatchQueue(ensembles, ctas_per_sm=1).run()
    torch.cuda.synchronize()
    for e, w in zip(ensembles, want):
        assert np.abs(w).min() > 0
        assert rel_l2(e.power().cpu().numpy(), w) <= 1e-5


@pytest.mark.parametrize("frames,shift", [(15, 0), (15, 1), (33, 0), (16, 1)])
def test_last_sample_keeps_the_next_slab_out(frames, shift):
    """A tap on a slab's last sample weighs the row behind it by zero: that row is zeros, not
    the next slab's samples (NaN here, of an angle whose window no voxel reaches)."""
    ns = 65
    rc = np.ones((ns, 1, 2, frames), np.complex64)
    rc[:, :, 1] = np.nan
    scan = np.array([[0.0, 2.0**-8, 0.0]], np.float32)  # delay 2^-17 s: sample 128 - 64, the last
    zero = np.zeros(1, np.float32)
    starts = np.array([64 * 2.0**-24, 1.0], np.float32)
    pd, iq = _reconstruct(rc, np.zeros_like(rc), scan, zero, zero, np.zeros(2, np.float32), starts, None, 0, shift,
                          c=2.0**10, fs=2.0**24, fd=0.0)
    assert np.array_equal(iq[0, 0], np.ones(frames, np.complex64)) and pd[0] == 1.0


@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("frames", [26, 78])
def test_power_sums_keep_small_frames(method, frames):
    """One strong frame among ones, every product exact: an item's float64 mean is rounded once
    to float32 and added to the others' (few tiles: items of 13 to 16 frames), 2^-24 per item;
    XDoppler's hypotf adds up to 3 ulp.  A float32 sum over frames loses all but the strong one."""
    value = np.ones(frames, np.complex64)
    value[0] = 2.0**12
    rc = np.broadcast_to(value, (64, 1, 1, frames)).copy()
    cr = rc if method == 1 else np.zeros_like(rc)
    scan = np.array([[0.0, 3e-3, 0.0]], np.float32)
    zero = np.zeros(1, np.float32)
    start = np.array([2 * 3e-3 / C - 1e-6], np.float32)
    pd, _ = _reconstruct(rc, cr, scan, zero, zero, zero, start, None, method, 0, fd=0.0)
    want = (2.0**24 + frames - 1) / frames
    bound = -(-frames // 16) + (6 if method == 1 else 0)
    assert abs(float(pd[0]) - want) <= bound * 2.0**-24 * want


def test_two_threads_of_different_sizes():
    """Launches of one kernel that need different amounts of shared memory do not fail each other."""
    errors = []

    def work(frames):
        rng = np.random.default_rng(frames)
        shape = (8, 1, 1, frames)
        rc = torch.from_numpy(rng.normal(size=shape).astype(np.complex64).transpose(1, 2, 0, 3).copy()).cuda()
        zero = torch.zeros(3, dtype=torch.float32, device="cuda")
        scan = torch.tensor([[0.0, 3e-3, 0.0]], device="cuda")
        pd = torch.empty(2, dtype=torch.float32, device="cuda")
        work = torch.empty(_cuda_impl.workspace_bytes(1, 1, 1), dtype=torch.uint8, device="cuda")
        try:
            for _ in range(2000):
                _lib.call("rcabeam_ensemble_device", rc.data_ptr(), rc.data_ptr(), scan.data_ptr(), zero.data_ptr(),
                          zero.data_ptr(), zero.data_ptr(), zero.data_ptr(), pd.data_ptr(), None, None, None,
                          work.data_ptr(), 8, 1, 1, frames, 1, C, FS, FD, -1.0, 0, 2)
        except _lib.RcabeamCudaError as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(frames,)) for frames in (2, 16)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors
