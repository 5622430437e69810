"""Staged host copies (rcabeam_host_copy): chunk and thread remainders, read-only sources, concurrent callers."""

from __future__ import annotations

import threading

import numpy as np
import pytest
import torch

from rcabeam_b200 import _cuda_impl

pytestmark = pytest.mark.gpu
CHUNK = 2 << 20


@pytest.fixture(autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("needs CUDA")


@pytest.mark.parametrize("nbytes", [8, CHUNK - 8, CHUNK, CHUNK + 8, 16 * CHUNK, 16 * CHUNK + 8, 37 * CHUNK - 16])
def test_round_trip_is_exact(nbytes):
    host = np.random.default_rng(nbytes).integers(0, 255, nbytes, dtype=np.uint8)
    host.flags.writeable = False
    device = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    _cuda_impl._host_copy(host, device, True)
    assert np.array_equal(device.cpu().numpy(), host)
    back = np.zeros(nbytes, np.uint8)
    _cuda_impl._host_copy(back, device, False)
    assert np.array_equal(back, host)


def test_concurrent_uploads_from_two_threads():
    arrays = [np.random.default_rng(i).standard_normal((1 << 20) + i).astype(np.complex64) for i in range(2)]
    out = [None, None]

    def work(i):
        for _ in range(3):
            out[i] = _cuda_impl._to_device(arrays[i], torch.complex64)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for a, d in zip(arrays, out):
        assert np.array_equal(d.cpu().numpy(), a)


@pytest.mark.parametrize("voxels", [1000, 300_000, 700_000])
def test_wider_host_outputs_are_converted(voxels):
    rng = np.random.default_rng(voxels)
    rc, cr = ((rng.normal(size=(64, 2, 1, 2)) + 1j * rng.normal(size=(64, 2, 1, 2))).astype(np.complex64)
              for _ in range(2))
    scan = rng.uniform([-1e-3, 3e-3, -1e-3], [1e-3, 4e-3, 1e-3], (voxels, 3)).astype(np.float32)
    el, zero = np.array([-1e-4, 1e-4], np.float32), np.zeros(1, np.float32)
    start = np.array([2 * 3e-3 / 1540 - 0.3e-6], np.float32)
    results = []
    for real, cplx in ((np.float32, np.complex64), (np.float64, np.complex128)):
        pd, signal = np.zeros((voxels, 2), real), np.zeros((voxels, 2), cplx)
        _cuda_impl.ensemble_from_channels(rc, cr, scan, el, el, zero, start, pd, signal, None, 1540.0, 20e6, 5e6, -1.0,
                                          0, 2, False)
        results.append((pd, signal))
    (pd, signal), (pd64, signal64) = results
    assert np.abs(signal).max() > 0
    assert np.array_equal(pd64, pd) and np.array_equal(signal64, signal)


def test_concurrent_staged_copies():
    hosts = [np.random.default_rng(i).integers(0, 255, 9 * CHUNK + 8 * i, dtype=np.uint8) for i in range(2)]
    back = [np.zeros_like(h) for h in hosts]

    def work(i):
        device = torch.empty(hosts[i].nbytes, dtype=torch.uint8, device="cuda")
        for _ in range(3):
            _cuda_impl._host_copy(hosts[i], device, True)
            _cuda_impl._host_copy(back[i], device, False)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for h, b in zip(hosts, back):
        assert np.array_equal(b, h)
